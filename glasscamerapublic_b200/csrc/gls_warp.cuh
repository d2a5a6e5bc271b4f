// gls_warp.cuh — the pull-warp of registerAndFuse / registerImage
// (SURF.metal:489-538): a frame sampled at H (x, y), exact bilinear
// interpolation, clamp-to-edge. One IEEE rounding per operation, so every
// caller gets the same bits.
#pragma once

#include <type_traits>

#include "gls_common.cuh"
#include "gls_fmath.h"

namespace gls {

template <class S>
__device__ __forceinline__ float4 rd4(const S* p) {
    if constexpr (std::is_same<S, float>::value) {
        return __ldg(reinterpret_cast<const float4*>(p));
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
}

__device__ __forceinline__ float lerp_(float a, float b, float t) {
    return glsm::fadd(a, glsm::fmul(t, glsm::fsub(b, a)));
}

// the four texels around H (x, y) and the interpolation weights
struct WarpPos {
    int xa, xb, ya, yb;
    float ax, ay;
};

__device__ __forceinline__ WarpPos warp_pos(const float (&H)[9], int x, int y, int iw, int ih) {
    using namespace glsm;
    const float fx = float(x), fy = float(y);
    const float u = fadd(fadd(fmul(H[0], fx), fmul(H[1], fy)), H[2]);
    const float v = fadd(fadd(fmul(H[3], fx), fmul(H[4], fy)), H[5]);
    const float ww = fadd(fadd(fmul(H[6], fx), fmul(H[7], fy)), H[8]);
    const float xx = fminf(fmaxf(fdiv(u, ww), -1.0f), float(iw));
    const float yy = fminf(fmaxf(fdiv(v, ww), -1.0f), float(ih));
    const float x0f = floorf(xx), y0f = floorf(yy);
    const int x0 = int(x0f), y0 = int(y0f);
    return {min(max(x0, 0), iw - 1), min(max(x0 + 1, 0), iw - 1), min(max(y0, 0), ih - 1), min(max(y0 + 1, 0), ih - 1),
            fsub(xx, x0f), fsub(yy, y0f)};
}

template <class S>
__device__ __forceinline__ float4 warp_sample(const S* in, size_t pitch, const WarpPos& q) {
    const S *ra = in + size_t(q.ya) * pitch, *rb = in + size_t(q.yb) * pitch;
    const float4 p00 = rd4(ra + 4 * q.xa), p10 = rd4(ra + 4 * q.xb);
    const float4 p01 = rd4(rb + 4 * q.xa), p11 = rd4(rb + 4 * q.xb);
    return make_float4(lerp_(lerp_(p00.x, p10.x, q.ax), lerp_(p01.x, p11.x, q.ax), q.ay),
                       lerp_(lerp_(p00.y, p10.y, q.ax), lerp_(p01.y, p11.y, q.ax), q.ay),
                       lerp_(lerp_(p00.z, p10.z, q.ax), lerp_(p01.z, p11.z, q.ax), q.ay),
                       lerp_(lerp_(p00.w, p10.w, q.ax), lerp_(p01.w, p11.w, q.ax), q.ay));
}

}  // namespace gls
