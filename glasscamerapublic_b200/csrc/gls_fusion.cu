// gls_fusion.cu — pyramid burst fusion (gls_fuse_pyramid).
//
// The reference declares a pyramid fusion API but has no live
// implementation (pyramid_processor.hpp:51-55, 64-70 are commented out); its
// burst driver fuses by registerAndFuse, a running mean of pull-warped
// frames (SURF.metal:489-516, pyramidFusion.cpp:343-345). This is the
// library's own design, built to reduce to that mean:
//   * every frame is pull-warped into the reference frame (registerImage);
//   * each warped frame is decomposed into a Laplacian pyramid with the
//     denoiser's own operators: 4-tap bilinear box down-sampling
//     (downsampleImageXYZ, demosaic.metal:886-920) and the reconstruct
//     step's bilinear up-sampling (subtractNoiseImage, :922-959);
//   * per level and pixel, frames are averaged with weights
//     w = exp(-robustness |band - band_ref|^2) (the reference frame has
//     weight 1); robustness 0 gives uniform weights;
//   * the fused pyramid is collapsed with the same up-sampling.
// The operators are linear, so with uniform weights the result is the flat
// mean of the warped frames (up to float rounding): registerAndFuse's output.
#include <algorithm>
#include <cmath>

#include "gls_common.cuh"
#include "gls_devbuf.h"
#include "gls_kernels.h"
#include "gls_warp.cuh"

namespace gls {

// Frames are fused in groups: the reference frame and up to kGroup - 1
// others. A group runs one launch per level for all of its frames, so a
// level's weighted sums stay in registers from the first frame to the last,
// and the level's fused band is collapsed onto the coarser result in the same
// kernel. The warped level-0 images never reach HBM: the pass that builds
// level 1 and the level-0 pass each warp the frames they read. A burst of up
// to kGroup frames (the usual one) is one group; longer bursts carry the sums
// from group to group in HBM.
//
// What bounds it, 8 x 4032x3024 FP16 frames, 5 levels, robust weights: the
// warps' and samplings' arithmetic (issue slots), not HBM: the frames are read
// twice and level 1 (49 MB a frame) is written once and read once. Measured:
// 1.26 ms a burst (level 1 0.38 ms at 78% of the issue slots, level 0 0.6 at 67%,
// the middle levels' passes 0.11 + 0.2 ms, near HBM / L2 rates), 3.28 ms with
// a launch per frame and level and every warped image and sum in HBM.
constexpr int kGroup = 8;

struct FuseFrame {
    const void* p;
    int pitch;  // elements
    int iw, ih;
    int half;   // F16 texels (else F32)
    int plain;  // warp3's short form holds for every pixel
    float H[9];
};
struct FuseFrames {
    FuseFrame f[kGroup];
};

// an RGB value as a packed FP32 pair and a scalar: an operation on it issues
// two instructions instead of three
struct Rgb {
    float2 xy;
    float z;
};
__device__ __forceinline__ float2 fma2f(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ Rgb sub(const Rgb& a, const Rgb& b) {
    return {fma2f(b.xy, make_float2(-1.f, -1.f), a.xy), a.z - b.z};
}
__device__ __forceinline__ Rgb axpy(float t, const Rgb& a, const Rgb& b) {  // t a + b
    return {fma2f(make_float2(t, t), a.xy, b.xy), fmaf(t, a.z, b.z)};
}
__device__ __forceinline__ Rgb mix(const Rgb& a, const Rgb& b, float t) { return axpy(t, sub(b, a), a); }

__device__ __forceinline__ Rgb rgb_at(const __half* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    return {__half22float2(*reinterpret_cast<const __half2*>(&u.x)),
            __low2float(*reinterpret_cast<const __half2*>(&u.y))};
}
__device__ __forceinline__ Rgb rgb_at(const float* p) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    return {make_float2(v.x, v.y), v.z};
}

// Bilinear sample at texel position (sx, sy) in [0, iw - 1] x [0, ih - 1],
// which gives what clamp-to-edge reads give outside: on the last column and row
// both texels are the last one.
template <class S>
__device__ __forceinline__ Rgb texel_mix(const FuseFrame& f, float sx, float sy) {
    const int x0 = int(sx), y0 = int(sy);
    const float ax = sx - float(x0), ay = sy - float(y0);
    const S* p0 = static_cast<const S*>(f.p) + size_t(unsigned(y0)) * unsigned(f.pitch) + 4 * unsigned(x0);
    const S* p1 = p0 + (y0 < f.ih - 1 ? unsigned(f.pitch) : 0u);
    const unsigned dx = x0 < f.iw - 1 ? 4u : 0u;
    return mix(mix(rgb_at(p0), rgb_at(p0 + dx), ax), mix(rgb_at(p1), rgb_at(p1 + dx), ax), ay);
}

// Frame f pull-warped at the N positions (x[k], y[k]) of the reference frame.
// The numerators and denominators are registerImage's, rounding for rounding.
// Where the host has shown the denominator to stay within (2^-10, 2^40) and
// the numerators to stay below 2^80 (every usual homography), a quotient is the
// approximate reciprocal's product corrected once by its remainder (Newton's
// iteration for the quotient): the division's result but for ties within the
// last 2^-22 of an ulp, in 7 instructions for the two quotients instead of
// two divisions' 24. All positions come before the first texel, so the
// texels of all N samples are in flight together. Other frames (a single row
// or column, a vanishing line through the image) take registerImage's form.
// HALF: FP16 frames all; else by the frame's own flag.
template <int N, bool HALF>
__device__ __forceinline__ void warp3(const FuseFrame& f, const int (&x)[N], const int (&y)[N], Rgb (&out)[N]) {
    using namespace glsm;
    if (!f.plain) {
#pragma unroll
        for (int k = 0; k < N; k++) {
            const WarpPos q = warp_pos(f.H, x[k], y[k], f.iw, f.ih);
            const float4 v = HALF || f.half
                                 ? warp_sample(static_cast<const __half*>(f.p), f.pitch, q)
                                 : warp_sample(static_cast<const float*>(f.p), f.pitch, q);
            out[k] = {make_float2(v.x, v.y), v.z};
        }
        return;
    }
    float sx[N], sy[N];
#pragma unroll
    for (int k = 0; k < N; k++) {
        const float fx = float(x[k]), fy = float(y[k]);
        const float u = fadd(fadd(fmul(f.H[0], fx), fmul(f.H[1], fy)), f.H[2]);
        const float v = fadd(fadd(fmul(f.H[3], fx), fmul(f.H[4], fy)), f.H[5]);
        const float w = fadd(fadd(fmul(f.H[6], fx), fmul(f.H[7], fy)), f.H[8]);
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(w));
        sx[k] = fmul(u, r);
        sy[k] = fmul(v, r);
        sx[k] = fmaf(fmaf(-sx[k], w, u), r, sx[k]);
        sy[k] = fmaf(fmaf(-sy[k], w, v), r, sy[k]);
        sx[k] = fminf(fmaxf(sx[k], 0.f), float(f.iw - 1));
        sy[k] = fminf(fmaxf(sy[k], 0.f), float(f.ih - 1));
    }
    if (HALF || f.half) {
#pragma unroll
        for (int k = 0; k < N; k++) out[k] = texel_mix<__half>(f, sx[k], sy[k]);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) out[k] = texel_mix<float>(f, sx[k], sy[k]);
    }
}

// the four texels and weights of a bilinear sample at texel position (u, v)
struct Bilin {
    int x0, x1, y0, y1;
    float ax, ay;
};
__device__ __forceinline__ Bilin bilin_at(float u, float v, int w, int h) {
    const float fu = floorf(u), fv = floorf(v);
    const int xi = int(fu), yi = int(fv);
    return {clampi(xi, 0, w - 1), clampi(xi + 1, 0, w - 1), clampi(yi, 0, h - 1), clampi(yi + 1, 0, h - 1), u - fu,
            v - fv};
}
__device__ __forceinline__ Rgb rgb_at(const float4* p) { return rgb_at(reinterpret_cast<const float*>(p)); }
__device__ __forceinline__ Rgb sample3(const float4* c, int cw, const Bilin& b) {
    const float4 *r0 = c + size_t(b.y0) * cw, *r1 = c + size_t(b.y1) * cw;
    return mix(mix(rgb_at(r0 + b.x0), rgb_at(r0 + b.x1), b.ax), mix(rgb_at(r1 + b.x0), rgb_at(r1 + b.x1), b.ax), b.ay);
}

// downsampleImageXYZ (demosaic.metal:886-920): the mean of four bilinear
// samples at (x r - 0.5, (x + 1) r - 0.5) in each direction. Neighbouring
// pixels share their samples, so a warp takes a strip of 31 columns: lane i
// samples column x0 + i of sample row k once, pairs of lanes and of
// successive rows are added. Each sample, and each texel under it, is formed
// once (1.03 x (rows + 1) / rows with the strip's edges) instead of four
// times, without shared memory. texels(xa, xb, ya, yb, t) reads the finer
// image at (xa, ya), (xb, ya), (xa, yb), (xb, yb).
constexpr int FD_COLS = 31;

template <int UNROLL, class Texels>
__device__ __forceinline__ void down_strip(float rx, float ry, int w, int h, int ow, int oh, int rows,
                                           float4* __restrict__ out, Texels&& texels) {
    const int lane = threadIdx.x, x = blockIdx.x * FD_COLS + lane;
    const int y0 = (blockIdx.y * blockDim.y + threadIdx.y) * rows;
    if (y0 >= oh) return;  // warp-uniform
    const float u = __fsub_rn(__fmul_rn(float(x), rx), 0.5f);
    const float fu = floorf(u), ax = u - fu;
    const int xa = clampi(int(fu), 0, w - 1), xb = clampi(int(fu) + 1, 0, w - 1);
    const int yn = min(rows, oh - y0);
    Rgb prev = {make_float2(0.f, 0.f), 0.f};
#pragma unroll UNROLL
    for (int k = 0; k <= yn; k++) {
        const float v = __fsub_rn(__fmul_rn(float(y0 + k), ry), 0.5f);
        const float fv = floorf(v);
        const int ya = clampi(int(fv), 0, h - 1), yb = clampi(int(fv) + 1, 0, h - 1);
        Rgb q[4];
        texels(xa, xb, ya, yb, q);
        const Rgb s = mix(mix(q[0], q[1], ax), mix(q[2], q[3], ax), v - fv);
        const Rgb t = {make_float2(s.xy.x + __shfl_down_sync(0xffffffffu, s.xy.x, 1),
                                   s.xy.y + __shfl_down_sync(0xffffffffu, s.xy.y, 1)),
                       s.z + __shfl_down_sync(0xffffffffu, s.z, 1)};
        if (k > 0 && lane < FD_COLS && x < ow)
            out[size_t(y0 + k - 1) * ow + x] =
                make_float4(0.25f * (prev.xy.x + t.xy.x), 0.25f * (prev.xy.y + t.xy.y), 0.25f * (prev.z + t.z), 0.f);
        prev = t;
    }
}

// Level 1 of the frames [first, first + gridDim.z) straight from the input
// frames: the texels are warped as the strip reads them
template <bool HALF>
__global__ void __launch_bounds__(256) k_fuse_level1(FuseFrames fr, int first, int W, int H, float4* __restrict__ out,
                                                     size_t out_stride, int w1, int h1, float rx, float ry, int rows) {
    const FuseFrame& f = fr.f[first + blockIdx.z];
    down_strip<1>(rx, ry, W, H, w1, h1, rows, out + blockIdx.z * out_stride,
                  [&](int xa, int xb, int ya, int yb, Rgb (&t)[4]) {
                      const int x[4] = {xa, xb, xa, xb}, y[4] = {ya, ya, yb, yb};
                      warp3<4, HALF>(f, x, y, t);
                  });
}

// the next coarser level of gridDim.z frames
__global__ void __launch_bounds__(256) k_fuse_down(const float4* __restrict__ in, size_t in_stride, int w, int h,
                                                   float4* __restrict__ out, size_t out_stride, int ow, int oh,
                                                   float rx, float ry, int rows) {
    const float4* src = in + blockIdx.z * in_stride;
    down_strip<4>(rx, ry, w, h, ow, oh, rows, out + blockIdx.z * out_stride,
                  [&](int xa, int xb, int ya, int yb, Rgb (&t)[4]) {
                      const float4 *ra = src + size_t(ya) * w, *rb = src + size_t(yb) * w;
                      t[0] = rgb_at(ra + xa);
                      t[1] = rgb_at(ra + xb);
                      t[2] = rgb_at(rb + xa);
                      t[3] = rgb_at(rb + xb);
                  });
}

struct FuseLevelArgs {
    int w, h, cw, ch;  // level and next-coarser sizes (cw = 0: coarsest level)
    float rx, ry;
    const float4 *g, *gc;        // this level and the coarser one, frame k at k * stride (level 0: no g)
    size_t g_stride, gc_stride;
    const float4* coarse;        // collapsed coarser level
    float4* acc;                 // sums carried between groups (null: one group)
    int n;                       // frames of the group, the reference (0) included
    int first_group, last_group;
    float robustness;
    void* out;                   // the fused level: float4 (scratch, level 0 included) or the caller's view
    size_t out_pitch;            // pixels
};

// One level of a group: every frame's band (its Gaussian level minus the
// up-sampled coarser one) into the weighted sums, in frame order, then, in
// the last group, the weighted mean plus the up-sampled coarser result. A
// thread takes the rows 2t - 1 and 2t: at a ratio of 2 both interpolate
// between the same two coarse rows, so the four coarse texels and their
// horizontal interpolation are shared; rows whose coarse rows differ (odd
// sizes) read their own.
// LEVEL0 warps the frames (HALF as in warp3); O: the output's element type.
// Four blocks an SM (64 registers): 1250 us a burst against 1404 with three
// at level 0 and 1449 to 1812 with two or four frames unrolled, which cost
// more occupancy than they add loads in flight.
template <bool LEVEL0, bool HALF, class O>
__global__ void __launch_bounds__(256, 4) k_fuse_level(FuseLevelArgs a, FuseFrames fr) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= a.w || 2 * t - 1 >= a.h) return;
    const int y[2] = {max(2 * t - 1, 0), min(2 * t, a.h - 1)};  // row -1 and row h: computed, not stored
    const int cw = max(a.cw, 1), ch = max(a.ch, 1);
    const float u = (float(x) + 0.5f) * a.rx - 0.5f;
    const Bilin b0 = bilin_at(u, (float(y[0]) + 0.5f) * a.ry - 0.5f, cw, ch);
    const Bilin b1 = bilin_at(u, (float(y[1]) + 0.5f) * a.ry - 0.5f, cw, ch);
    const bool shared_rows = b0.y0 == b1.y0 && b0.y1 == b1.y1;  // uniform over a row of threads
    auto up2 = [&](const float4* c, Rgb (&r)[2]) {
        const float4 *r0 = c + size_t(b0.y0) * cw, *r1 = c + size_t(b0.y1) * cw;
        const Rgb top = mix(rgb_at(r0 + b0.x0), rgb_at(r0 + b0.x1), b0.ax);
        const Rgb bot = mix(rgb_at(r1 + b0.x0), rgb_at(r1 + b0.x1), b0.ax);
        r[0] = mix(top, bot, b0.ay);
        r[1] = shared_rows ? mix(top, bot, b1.ay) : sample3(c, cw, b1);
    };
    const size_t i[2] = {size_t(y[0]) * a.w + x, size_t(y[1]) * a.w + x};
    auto bands = [&](int k, Rgb (&b)[2]) {
        if constexpr (LEVEL0) {
            const int xs[2] = {x, x};
            warp3<2, HALF>(fr.f[k], xs, y, b);
        } else {
            b[0] = rgb_at(a.g + size_t(k) * a.g_stride + i[0]);
            b[1] = rgb_at(a.g + size_t(k) * a.g_stride + i[1]);
        }
        if (a.cw > 0) {
            Rgb r[2];
            up2(a.gc + size_t(k) * a.gc_stride, r);
            b[0] = sub(b[0], r[0]);
            b[1] = sub(b[1], r[1]);
        }
    };
    Rgb rb[2], c[2];
    float cs[2];  // the sums of the weights
    bands(0, rb);
#pragma unroll
    for (int e = 0; e < 2; e++) {
        c[e] = rb[e];
        cs[e] = 1.f;
        if (!a.first_group) {
            const float4 v = a.acc[i[e]];
            c[e] = {make_float2(v.x, v.y), v.z};
            cs[e] = v.w;
        }
    }
#pragma unroll 1
    for (int k = 1; k < a.n; k++) {
        Rgb b[2];
        bands(k, b);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float w = 1.f;
            if (a.robustness > 0.f) {
                const Rgb d = sub(b[e], rb[e]);
                w = expf(-a.robustness * (d.xy.x * d.xy.x + d.xy.y * d.xy.y + d.z * d.z));
            }
            c[e] = axpy(w, b[e], c[e]);
            cs[e] += w;
        }
    }
    const bool store[2] = {t > 0, 2 * t < a.h};
    if (!a.last_group) {
#pragma unroll
        for (int e = 0; e < 2; e++)
            if (store[e]) a.acc[i[e]] = make_float4(c[e].xy.x, c[e].xy.y, c[e].z, cs[e]);
        return;
    }
    Rgb r[2] = {};
    if (a.cw > 0) up2(a.coarse, r);
#pragma unroll
    for (int e = 0; e < 2; e++)
        if (store[e])
            st4<O>(static_cast<O*>(a.out) + (size_t(y[e]) * a.out_pitch + x) * 4,
                   f4{c[e].xy.x / cs[e] + r[e].xy.x, c[e].xy.y / cs[e] + r[e].xy.y, c[e].z / cs[e] + r[e].z, 0.f});
}

template <class O>
__global__ void k_fuse_store(const float4* in, int w, int h, O* out, size_t pitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float4 v = in[size_t(y) * w + x];
    st4<O>(out + size_t(y) * pitch + size_t(x) * 4, f4{v.x, v.y, v.z, v.w});
}

// scratch kept by the registration context between calls: the Gaussian
// levels 1.. of a group's frames, the collapsed levels, and for bursts of
// more than one group the carried sums. col[0] is used only when the output
// overlaps an input frame.
struct FusionScratch {
    DevBuf g[GLS_MAX_LEVELS], acc[GLS_MAX_LEVELS], col[GLS_MAX_LEVELS];
    ~FusionScratch() {
        for (int l = 0; l < GLS_MAX_LEVELS; l++) {
            g[l].release();
            acc[l].release();
            col[l].release();
        }
    }
};

FusionScratch* fusion_scratch_new() { return new FusionScratch(); }
void fusion_scratch_delete(FusionScratch* f) { delete f; }

// the checks that registerImage makes of each input
static gls_status fuse_frame(const gls_image_view& v, const float* H, int w, int h, FuseFrame& f) {
    if (!v.data) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (v.channels != 4 || (v.dtype != GLS_F32 && v.dtype != GLS_F16))
        return set_error(GLS_ERR_INVALID_ARG, "input must be RGBA GLS_F32 or GLS_F16");
    if (v.width < 1 || v.height < 1) return set_error(GLS_ERR_INVALID_ARG, "empty image");
    const size_t es = v.dtype == GLS_F32 ? 4 : 2;
    const size_t stride = v.stride_bytes ? v.stride_bytes : size_t(v.width) * 4 * es;
    if (stride % (4 * es) || (reinterpret_cast<uintptr_t>(v.data) % (4 * es)))
        return set_error(GLS_ERR_INVALID_ARG, "pixel rows must be aligned to whole RGBA pixels");
    f.p = v.data;
    f.pitch = int(stride / es);
    f.iw = v.width;
    f.ih = v.height;
    f.half = v.dtype == GLS_F16;
    for (int k = 0; k < 9; k++) f.H[k] = H[k];
    // warp3's short form: a denominator within (2^-10, 2^40) at the w x h
    // output's corners (it is linear between them) and bounded numerators
    bool plain = f.iw >= 2 && f.ih >= 2;
    for (int c = 0; c < 4; c++) {
        const double x = c & 1 ? w - 1 : 0, y = c & 2 ? h - 1 : 0;
        const double d = double(H[6]) * x + double(H[7]) * y + double(H[8]);
        plain = plain && d > 0x1p-10 && d < 0x1p40;
    }
    // its terms below 2^6, so that its FP32 rounding is below 2^-15
    const float lim = 0x1p6f / float(std::max(w, h));
    for (int k = 0; k < 9; k++) plain = plain && std::fabs(H[k]) < (k < 6 ? 0x1p60f : k < 8 ? lim : 0x1p6f);
    f.plain = plain;
    return GLS_OK;
}

// fn(bool constant HALF) for a group's texel format (warp3)
template <class Fn>
static void by_format(bool half, Fn&& fn) {
    if (half) fn(std::true_type{});
    else fn(std::false_type{});
}

static bool overlaps(const gls_image_view& a, const gls_image_view& b) {
    auto end = [](const gls_image_view& v) {
        const size_t row = size_t(v.width) * 4 * (v.dtype == GLS_F32 ? 4 : 2);
        return uintptr_t(v.data) + (v.stride_bytes ? v.stride_bytes : row) * size_t(v.height - 1) + row;
    };
    return uintptr_t(a.data) < end(b) && uintptr_t(b.data) < end(a);
}

gls_status fuse_pyramid_impl(FusionScratch* F, const gls_image_view* frames, int n, const float* H, int levels,
                             float robustness, gls_image_view* out, cudaStream_t s) {
    static const float I[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    const int W = frames[0].width, Hh = frames[0].height;
    const int slots = std::min(n, kGroup), groups = n > kGroup ? (n - 2) / (kGroup - 1) + 1 : 1;
    bool overlap = false;
    for (int f = 0; f < n; f++) {  // every frame is checked before any work is queued
        FuseFrame t;
        GLS_TRY(fuse_frame(frames[f], f == 0 ? I : H + size_t(f) * 9, W, Hh, t));
        overlap = overlap || overlaps(frames[f], *out);
    }
    auto px = [&](int l) { return size_t(W >> l) * (Hh >> l); };
    for (int l = 0; l < levels; l++) {
        if (l > 0) GLS_TRY(F->g[l].ensure(px(l) * slots * 16));
        if (l > 0 || overlap) GLS_TRY(F->col[l].ensure(px(l) * 16));
        if (groups > 1) GLS_TRY(F->acc[l].ensure(px(l) * 16));
    }
    auto g = [&](int l, int k) { return static_cast<float4*>(F->g[l].p) + px(l) * k; };
    auto grid = [](int w, int h) { return dim3((w + 31) / 32, (h + 7) / 8); };
    auto grid2 = [](int w, int h) { return dim3((w + 31) / 32, (h / 2 + 8) / 8); };  // h / 2 + 1 row pairs
    const dim3 blk(32, 8);
    const size_t es = out->dtype == GLS_F32 ? 4 : 2;
    const size_t pitch = (out->stride_bytes ? out->stride_bytes : size_t(W) * 4 * es) / es;
    for (int grp = 0; grp < groups; grp++) {
        // the group's frames: slot 0 the reference, then frames f0 ..
        const int f0 = 1 + grp * (kGroup - 1), cnt = 1 + std::min(kGroup - 1, n - f0);
        FuseFrames fr{};
        for (int k = 0; k < cnt; k++) {
            const int f = k == 0 ? 0 : f0 + k - 1;
            GLS_TRY(fuse_frame(frames[f], f == 0 ? I : H + size_t(f) * 9, W, Hh, fr.f[k]));
        }
        bool halves = true;
        for (int k = 0; k < cnt; k++) halves = halves && fr.f[k].half;
        const int k0 = grp == 0 ? 0 : 1;  // the reference's levels are built once
        for (int l = 1; l < levels; l++) {
            const int w = W >> (l - 1), h = Hh >> (l - 1), ow = W >> l, oh = Hh >> l;
            const float rx = float(w) / float(ow), ry = float(h) / float(oh);
            // 16 rows a strip (6% of the samples formed twice), 4 where
            // the level has fewer strips than the GPU has warp slots
            const int rows = size_t(ow) * oh * (cnt - k0) >= (size_t(1) << 22) ? 16 : 4;
            const dim3 gs((ow + FD_COLS - 1) / FD_COLS, (oh + 8 * rows - 1) / (8 * rows), cnt - k0);
            if (l > 1)
                k_fuse_down<<<gs, blk, 0, s>>>(g(l - 1, k0), px(l - 1), w, h, g(l, k0), px(l), ow, oh, rx, ry, rows);
            else
                by_format(halves, [&](auto half) {
                    k_fuse_level1<half.value><<<gs, blk, 0, s>>>(fr, k0, W, Hh, g(1, k0), px(1), ow, oh, rx, ry, rows);
                });
        }
        for (int l = levels - 1; l >= 0; l--) {
            FuseLevelArgs a{};
            a.w = W >> l;
            a.h = Hh >> l;
            if (l + 1 < levels) {
                a.cw = W >> (l + 1);
                a.ch = Hh >> (l + 1);
                a.rx = float(a.cw) / float(a.w);
                a.ry = float(a.ch) / float(a.h);
                a.gc = g(l + 1, 0);
                a.gc_stride = px(l + 1);
                a.coarse = static_cast<const float4*>(F->col[l + 1].p);
            }
            a.acc = static_cast<float4*>(F->acc[l].p);
            a.n = cnt;
            a.first_group = grp == 0;
            a.last_group = grp + 1 == groups;
            a.robustness = robustness;
            const bool to_caller = l == 0 && !overlap;
            a.out = to_caller ? out->data : F->col[l].p;
            a.out_pitch = to_caller ? pitch / 4 : size_t(a.w);
            if (l > 0) {
                a.g = g(l, 0);
                a.g_stride = px(l);
                k_fuse_level<false, false, float><<<grid2(a.w, a.h), blk, 0, s>>>(a, fr);
            } else {
                by_format(halves, [&](auto half) {
                    if (to_caller && out->dtype == GLS_F16)
                        k_fuse_level<true, half.value, __half><<<grid2(a.w, a.h), blk, 0, s>>>(a, fr);
                    else
                        k_fuse_level<true, half.value, float><<<grid2(a.w, a.h), blk, 0, s>>>(a, fr);
                });
            }
        }
    }
    if (overlap) {
        const float4* c = static_cast<const float4*>(F->col[0].p);
        if (out->dtype == GLS_F32)
            k_fuse_store<float><<<grid(W, Hh), blk, 0, s>>>(c, W, Hh, static_cast<float*>(out->data), pitch);
        else
            k_fuse_store<__half><<<grid(W, Hh), blk, 0, s>>>(c, W, Hh, static_cast<__half*>(out->data), pitch);
    }
    GLS_CUDA(cudaGetLastError());
    return GLS_OK;
}

}  // namespace gls
