// What both fine kernels share (fine.cu, fine_paths.cu): the decoded paints'
// layout, sample_gradient and the image patterns, and the rows a segment
// crosses.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "kernels.h"

namespace tk {
namespace {

using namespace tkd;

constexpr uint32_t kClipSpill = 28;
constexpr uint32_t kGroupDepth = 6;
constexpr uint32_t kGroupLocal = 2;  // FINE_LOCAL_GROUP_DEPTH (fine/constants.hlsli:11)
constexpr uint32_t kGradient = 0xFFFFFFFFu;
constexpr uint32_t kGradParams = 24;
constexpr uint32_t kGradConst = 0, kGradLinear = 1, kGradRadial = 2, kGradPattern = 3;  // decoded kinds
constexpr uint32_t kGradBilinear = 1u << 16;  // pattern: bilinear sampling
constexpr uint32_t kGradDenOk = 1u << 16;    // linear: den > GRADIENT_FLOAT_EPSILON
constexpr uint32_t kGradASmall = 1u << 16;   // radial: |a| <= RADIAL_QUADRATIC_EPSILON
constexpr uint32_t kGradFast = 1u << 17;     // linear, radial: the divisor allows divide_by
constexpr uint32_t kGradIdentity = 1u << 19; // linear, radial: both transforms are the identity
constexpr uint32_t kGradRampOk = 1u << 18;   // linear, radial: the ramp has two texels or more, inside the brush words


__device__ __forceinline__ bool is_fill_like(uint32_t tag) {
    return tag == TK_PTCL_FILL || tag == TK_PTCL_BEGIN_CLIP || tag == TK_PTCL_BEGIN_OPACITY ||
           tag == TK_PTCL_BEGIN_BLEND || tag == TK_PTCL_PATH_GLYPH;
}

// Division by a divisor that many pixels share, from its rounded reciprocal:
// P. Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor (1990). q is within two units of a / b, each step's remainder is
// exact in one fused multiply-add, and the second correction rounds correctly,
// as long as nothing underflows or overflows: hence the ranges. 5 FMA-pipe
// operations, which also run as pairs, against 10 and a branch.
__device__ __forceinline__ bool divisor_is_plain(float b) { return fabsf(b) > 0x1p-40f && fabsf(b) < 0x1p40f; }
__device__ __forceinline__ bool dividend_is_plain(float a) { return fabsf(a) > 0x1p-60f && fabsf(a) < 0x1p60f; }
__device__ __forceinline__ float divide_by(float a, float b, float rcp_b) {
    float q = a * rcp_b;
    q = mad(mad(-q, b, a), rcp_b, q);
    return mad(mad(-q, b, a), rcp_b, q);
}

// extend_coord_i32 (shared/brush/pattern.hlsli:9-17) with
// euclidean_remainder_i32 (shared/integer.hlsli:5-9).
__device__ __forceinline__ uint32_t extend_coord(int32_t v, uint32_t size, uint32_t extend) {
    if (size <= 1u) return 0u;
    if (extend == TK_EXTEND_REPEAT || extend == TK_EXTEND_REFLECT) {
        const uint32_t period = size * (extend == TK_EXTEND_REFLECT ? 2u : 1u);
        const uint32_t mag = v < 0 ? 0u - uint32_t(v) : uint32_t(v), rem = mag % period;
        const uint32_t coord = v < 0 && rem != 0u ? period - rem : rem;
        return coord < size ? coord : period - coord - 1u;
    }
    return uint32_t(min(max(v, 0), int32_t(size) - 1));
}

// lerp_premul_u8 (shared/pixel.hlsli:55-62): one fused interpolation per channel.
__device__ __forceinline__ uint32_t lerp_premul_u8(uint32_t a, uint32_t b, float t) {
    uint32_t out = 0u;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float l = float((a >> (8 * c)) & 255u), r = float((b >> (8 * c)) & 255u);
        out |= f2u(clampf(mad(r - l, t, l) + 0.5f, 0.0f, 255.0f)) << (8 * c);
    }
    return out;
}

// The image pattern decoded in g / k at brush-space point (x, y):
// pattern_transform_component (shared/pattern_transform.hlsli:7-11) and
// sample_resource_pattern_texture (shared/brush/texture.hlsli:11-31). Float to
// integer conversions saturate and take NaN to 0. The bilinear, pad-extended
// form is the texture unit's filter in the reference (SampleLevel with
// clamp-to-edge addressing); here it is that filter computed exactly: texel
// centres at half-integers, f32 weights, one rounding to 8 bits.
__device__ __noinline__ uint32_t pattern_at(const Paint& P, const float* g, uint4 k, float x, float y) {
    const float bx = g[8] * y, by = g[9] * y;
    const float tx = ((mad(g[6], x, bx) + mad(g[8], y, -bx)) + g[10]) * g[12];
    const float ty = ((mad(g[7], x, by) + mad(g[9], y, -by)) + g[11]) * g[13];
    const uint32_t w = __float_as_uint(g[14]), h = __float_as_uint(g[15]), extend = k.w;
    const uint32_t* __restrict__ tex = P.texels + k.y;
    uint32_t color;
    if ((k.x & kGradBilinear) && extend == TK_EXTEND_PAD) {
        const float sx = clampf(tx, 0.0f, g[12]) - 0.5f, sy = clampf(ty, 0.0f, g[13]) - 0.5f;
        const float fx0 = floorf(sx), fy0 = floorf(sy), fx = sx - fx0, fy = sy - fy0;
        const int32_t ix = __float2int_rz(fx0), iy = __float2int_rz(fy0);
        const uint32_t x0 = uint32_t(min(max(ix, 0), int32_t(w) - 1)), x1 = uint32_t(min(max(ix + 1, 0), int32_t(w) - 1));
        const uint32_t y0 = uint32_t(min(max(iy, 0), int32_t(h) - 1)), y1 = uint32_t(min(max(iy + 1, 0), int32_t(h) - 1));
        const float4 tl = rgba8_to_unorm(__ldg(tex + uint64_t(y0) * w + x0)), tr = rgba8_to_unorm(__ldg(tex + uint64_t(y0) * w + x1));
        const float4 bl = rgba8_to_unorm(__ldg(tex + uint64_t(y1) * w + x0)), br = rgba8_to_unorm(__ldg(tex + uint64_t(y1) * w + x1));
        const float4 top = make_float4(mad(tr.x - tl.x, fx, tl.x), mad(tr.y - tl.y, fx, tl.y), mad(tr.z - tl.z, fx, tl.z),
                                       mad(tr.w - tl.w, fx, tl.w));
        const float4 bot = make_float4(mad(br.x - bl.x, fx, bl.x), mad(br.y - bl.y, fx, bl.y), mad(br.z - bl.z, fx, bl.z),
                                       mad(br.w - bl.w, fx, bl.w));
        color = unorm_to_rgba8(make_float4(mad(bot.x - top.x, fy, top.x), mad(bot.y - top.y, fy, top.y),
                                           mad(bot.z - top.z, fy, top.z), mad(bot.w - top.w, fy, top.w)));
    } else if (k.x & kGradBilinear) {
        const float sx = tx - 0.5f, sy = ty - 0.5f;
        const float fx0 = floorf(sx), fy0 = floorf(sy), fx = sx - fx0, fy = sy - fy0;
        const int32_t ix = __float2int_rz(fx0), iy = __float2int_rz(fy0);
        const int32_t jx = int32_t(uint32_t(ix) + 1u), jy = int32_t(uint32_t(iy) + 1u);
        const uint64_t r0 = uint64_t(extend_coord(iy, h, extend)) * w, r1 = uint64_t(extend_coord(jy, h, extend)) * w;
        const uint32_t c0 = extend_coord(ix, w, extend), c1 = extend_coord(jx, w, extend);
        const uint32_t top = lerp_premul_u8(__ldg(tex + r0 + c0), __ldg(tex + r0 + c1), fx);
        const uint32_t bot = lerp_premul_u8(__ldg(tex + r1 + c0), __ldg(tex + r1 + c1), fx);
        color = lerp_premul_u8(top, bot, fy);
    } else {
        const uint32_t c = extend_coord(__float2int_rz(floorf(tx)), w, extend);
        const uint32_t r = extend_coord(__float2int_rz(floorf(ty)), h, extend);
        color = __ldg(tex + uint64_t(r) * w + c);
    }
    return scale_premul_u8(color, k.z);
}

// sample_gradient at pixel centre (px, py) for the gradient decoded in g / k.
// IMG: whether image patterns can occur (only SDF draws carry them).
template <bool IMG>
__device__ __forceinline__ uint32_t gradient_at(const float* g, const uint4 k, const Paint& P, float px, float py) {
    const uint32_t code = k.x & 255u, extend = k.w;
    if (code == kGradConst) return k.y;
    const float x = mad(g[0], px, mad(g[2], py, g[4]));
    const float y = mad(g[1], px, mad(g[3], py, g[5]));
    if (IMG && code == kGradPattern) return pattern_at(P, g, k, x, y);
    const float tx = mad(g[6], x, mad(g[8], y, g[10]));
    const float ty = mad(g[7], x, mad(g[9], y, g[11]));
    float t = 0.0f;
    if (code == kGradLinear) {
        if (k.x & kGradDenOk) t = mad(tx - g[12], g[14], (ty - g[13]) * g[15]) / g[16];
    } else {
        const float qx = tx - g[12], qy = ty - g[13];
        const float b = -2.0f * mad(qx, g[14], mad(qy, g[15], g[16]));
        const float c = mad(qx, qx, mad(qy, qy, g[17]));
        const float dr = g[21], sr = g[22];
        bool has_t = false;
        if (k.x & kGradASmall) {
            if (fabsf(b) > RADIAL_QUADRATIC_EPSILON) {
                const float cand = -c / b;
                if (mad(cand, dr, sr) >= 0.0f) {
                    has_t = true;
                    t = cand;
                }
            }
        } else {
            const float disc = mad(b, b, g[19] * c);
            if (disc >= 0.0f) {
                const float root = sqrtf(disc);
                const float t0 = (-b - root) / g[20], t1 = (-b + root) / g[20];
                const bool v0 = mad(t0, dr, sr) >= 0.0f, v1 = mad(t1, dr, sr) >= 0.0f;
                if (v0) {
                    has_t = true;
                    t = v1 ? fmaxf(t0, t1) : t0;
                } else if (v1) {
                    has_t = true;
                    t = t1;
                }
            }
        }
        if (!has_t) return 0u;
    }
    return sample_ramp(P, k.y, k.z, t, extend);
}


// The rows a segment crosses, i.e. where segment_row_parts gives dy != 0:
// with lo < hi the segment's y extent, clamp(y - row, 0, 1) differs between
// its ends exactly for rows floor(lo) .. ceil(hi) - 1 (y - row is exact for y
// in [row, row + 1], and rounds to the same side of that interval otherwise).
__device__ __forceinline__ uint32_t crossed_rows(float p0y, float p1y) {
    const float lo = fminf(p0y, p1y), hi = fmaxf(p0y, p1y);
    if (!(lo < hi)) return 0u;
    const int32_t r0 = max(f2i(floorf(lo)), 0), r1 = min(f2i(ceilf(hi)) - 1, int32_t(TK_TILE_SIZE) - 1);
    if (r1 < r0) return 0u;
    return ((2u << r1) - 1u) & ~((1u << r0) - 1u);
}

}  // namespace
}  // namespace tk
