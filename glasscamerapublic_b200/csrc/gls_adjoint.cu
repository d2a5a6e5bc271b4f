// gls_adjoint.cu — the hand-written adjoint of the pyramid denoise and
// reconstruct (PyramidProcessor<levels>::denoise, pyramid_processor.cpp:96-172,
// and the output transform, raw_converter.cpp:219) on the FP32 path.
//
// Given the forward's retained planes (per level: the layer that block
// matching denoised, its gradient plane, the denoised result, the frozen
// PCA basis) and dL/d(output RGB) of an MSE loss, it returns dL/dtheta for
// the per-level parameters that enter the pyramid:
//   luma_l, chroma_l       DenoiseParameters::luma / chroma (demosaic.hpp:33-40)
//   A_Y, B_Y, A_C, B_C     the level's YCbCr NLF a[0], b[0], a[1] = a[2], b[1] = b[2]
// The PCA basis is held fixed (its dependence on theta is not differentiated).
//
// Reverse sweep, fine to coarse: out = M den_0; den_l = BM_l(layer_l);
// layer_l = SN_l(img_l, img_{l+1}, den_{l+1}) for l < L-1, and
// layer_{L-1} = img_{L-1}. The pyramid parameters reach the loss through
// den_{l+1}; the raw green NLF reaches it through the input pyramid
// img_{l+1} = down(img_l), img_0 = the despeckled front-end output, so the
// sweep also accumulates dL/d img_l and pushes it down to img_0.
//   * k_adj_head          dL/d den_0 = M^T 2 (out - target) / N, and the loss
//   * k_bm_bwd_record     per pixel, what block matching's transpose needs of
//                         it: from the forward's outputs and kernel norms
//   * k_bm_bwd            block matching transposed, each pixel as a window
//                         centre and as a neighbour q of every centre p whose
//                         window reads it (clamp-to-edge preimages included):
//                         dL/d(layer), dL/d(PCA coefficients), dL/dtheta
//   * k_pca_bwd           transpose of the 5x5 x 25x8 projection
//   * k_sn_bwd            subtractNoiseImage: dL/d(up-sampled den_{l+1}) and
//                         dL/dtheta through the sharpening gate
//   * k_up_bwd            transpose of the bilinear up-sampling (for the
//                         coarse denoised image, and with k_up_bwd_img for
//                         the coarse noisy image)
//   * k_down_bwd          transpose of the pyramid down-sampling: with the
//                         subtract-noise input terms, dL/d(level-0 image),
//                         which the raw front end's tangents
//                         (gls_front_jvp.cu) turn into dL/d(raw green NLF)
// Every reduction is per block and summed in block order: the gradient does
// not depend on scheduling.
#include <cfloat>
#include <type_traits>

#include "gls_common.cuh"
#include "gls_kernels.h"

namespace gls {

constexpr int AT_X = 32;  // adjoint tile width
constexpr int AH = 10;    // block-matching window radius

// offsets d in [-R, R] with clamp(p + d, 0, n - 1) == q
__device__ __forceinline__ bool preimage(int q, int p, int R, int n, int& lo, int& hi) {
    lo = q - p;
    hi = q - p;
    if (q == 0) lo = -R;
    if (q == n - 1) hi = R;
    lo = max(lo, -R);
    hi = min(hi, R);
    return lo <= hi;
}

__device__ __forceinline__ float sstep(float e0, float e1, float x, float* dx) {  // smoothstep and d/dx
    const float t = (x - e0) / (e1 - e0);
    if (t <= 0.f) {
        *dx = 0.f;
        return 0.f;
    }
    if (t >= 1.f) {
        *dx = 0.f;
        return 1.f;
    }
    *dx = 6.f * t * (1.f - t) / (e1 - e0);
    return t * t * (3.f - 2.f * t);
}

// Per-pixel scales of blockMatchingDenoiseImage (demosaic.metal:806-850)
// and their partial derivatives.
struct BmScales {
    float L, K1, K2;              // luma distance scale, chroma scales
    float dL_dsig0, dK1_dsig1, dK2_dsig2;
    float sig0, sig1, sig2;
};

__device__ __forceinline__ BmScales bm_scales(const AdjointLevelArgs& a, float y, float mag) {
    BmScales s;
    s.sig0 = sqrtf(a.var_a[0] + a.var_b[0] * y);
    s.sig1 = sqrtf(a.var_a[1] + a.var_b[1] * y);
    s.sig2 = sqrtf(a.var_a[2] + a.var_b[2] * y);
    const float dm0 = 1.f / (a.tm[0] * s.sig0), dm1 = 1.f / (a.tm[1] * s.sig1), dm2 = 1.f / (a.tm[2] * s.sig2);
    const float z = a.gradient_threshold * mag / s.sig0;
    float dedge_dz;
    const float edge = sstep(2.f, 16.f, z, &dedge_dz);
    const float den = 1.f + a.gradient_boost * edge;
    s.L = dm0 / den;
    // dL/dsig0 = -L / sig0 + dL/dedge * dedge/dz * dz/dsig0
    const float dL_dedge = -s.L * a.gradient_boost / den;
    s.dL_dsig0 = -s.L / s.sig0 + dL_dedge * dedge_dz * (-z / s.sig0);
    s.K1 = dm1 / a.chroma_boost;
    s.K2 = dm2 / a.chroma_boost;
    s.dK1_dsig1 = -s.K1 / s.sig1;
    s.dK2_dsig2 = -s.K2 / s.sig2;
    return s;
}

__device__ __forceinline__ float spatial_w(int i, int j) {
    const float d = 0.1f * sqrtf(float(i * i + j * j));
    return expf(-2.f * d * d);
}

__device__ __forceinline__ float ex2a(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

typedef unsigned long long u64;
__device__ __forceinline__ u64 pk2(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 up2(u64 r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Per pixel, what its pairs need of it (12 floats):
//   Y, kl, Cb, Cr | gY/ny, gY/ny (Y - Y_out), g . (chroma - chroma_out), - | g, K^2
// with kl = -2 log2(e) L^2, S = sqrt(2 log2 e), g = 4 / S (gCb, gCr)/nc and
// K = S (K1, K2). In these units, for a centre's tap of spatial weight s at
// coefficient distance d2, luma difference dY and chroma difference c:
// l = exp2(kl d2 + log2 S) is S times the luma weight, the chroma weight is
// cw = exp2(-l^2 - |K c|^2), and with w = s cw (g . (chroma + c - chroma_out)):
//   dL/dL      = -4 L / S   sum d2 E,   E = l (s gY (Y + dY - Y_out) - w l)
//   dL/dK1     = -K         sum w c^2   (each channel)
//   dL/dchroma =  1 / S     sum w c K^2    (of both ends; plus the mean's term)
//   dL/dpca    = -4 / S^3   sum kl E (q - p)   (of both ends)
// The differences from the outputs are taken relative to the centre, so that
// nothing cancels.
constexpr float kAdjS = 1.6986436005760381f, kAdjLog2S = 0.7643831864724489f;

__global__ void __launch_bounds__(256) k_bm_bwd_record(AdjointLevelArgs a) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= a.w || y >= a.h) return;
    const size_t pi = size_t(y) * a.w + x;
    const float4 in = *reinterpret_cast<const float4*>(a.layer + pi * 4);
    const float2 gr = *reinterpret_cast<const float2*>(a.grad + pi * 2);
    const BmScales S = bm_scales(a, in.x, sqrtf(gr.x * gr.x + gr.y * gr.y));
    const float4 dv = *reinterpret_cast<const float4*>(a.den + pi * 4);
    const float* g = a.g_den + pi * 3;
    const float nc = a.nc[pi], k = 4.f / kAdjS;
    float4* rec = reinterpret_cast<float4*>(a.rec + pi * 12);
    rec[0] = make_float4(in.x, -kAdjS * kAdjS * S.L * S.L, in.y, in.z);
    const float gY = g[0] / dv.w, g1 = k * (g[1] / nc), g2 = k * (g[2] / nc);
    const float K1 = kAdjS * S.K1, K2 = kAdjS * S.K2;
    rec[1] = make_float4(gY, gY * (in.x - dv.x), fmaf(g1, in.y - dv.y, g2 * (in.z - dv.z)), 0.f);
    rec[2] = make_float4(g1, g2, K1 * K1, K2 * K2);
}

// Block matching transposed: every pixel x against every pixel y of the
// 21 x 21 box around it, x as the centre that reads y and x as the neighbour
// that the centre y reads. Both weights take the same coefficient distance,
// and both gradients of x's coefficients run along y - x: one pass over the
// pairs does both.
//
// A pixel at the image border is read through several taps that clamp onto it.
// All terms are linear in the spatial weight, so such a pair takes the sum of
// its taps' weights: a product of a column and a row table, used by the blocks
// whose box touches the border (0 for positions outside the image).
//
// What bounds it: the FMA pipe and the MUFU together (69 FP32 operations and 4
// ex2 a pair) and, with one pixel a thread, the 80 bytes of a pair's other
// pixel (20 shared-memory wavefronts for a warp); a thread takes two vertically
// adjacent pixels, whose windows share 20 of 22 rows. A block's 12 warps take
// 32 x 24 pixels (183 KB of staging, one block an SM), or, KS = 4, 8 warps take
// 32 x 4 pixels with each window's rows dealt to four warps, for levels too
// small to fill the chip. 2048x1536: 3.87 ms (8 warps 4.05, 16 warps 3.92),
// where a pass for the centres and one for the neighbours took 3.49 + 4.39;
// 128x96: 45 us for 75 + 308.
template <int KS>
struct BwdTile {
    static constexpr int WARPS = KS == 1 ? 12 : 8, THREADS = 32 * WARPS;
    static constexpr int ROWS = 2 * WARPS / KS, W = AT_X + 2 * AH, H = ROWS + 2 * AH;
    struct Smem {
        float4 v[5][H * W];  // the record, pca 0..3, pca 4..7
        union {
            float2 sw[22][21];  // the weights of box rows j and j - 1
            struct {            // weights of a pair by offset, x as the centre / as the neighbour
                float cx[AT_X][21], nx[AT_X][21];
                float2 y[ROWS][21];
            } b;
        };
    };
};

struct BwdPix {
    u64 n[4], nc;  // minus the coefficients, minus the chroma
    float Y, kl, gY, gYd, gcd, g1, g2, K1, K2;  // the record
    // sums
    u64 p[4];
    float E, luma, c1, c2, cc1, cc2, mean1, mean2, n1, n2;
};

__device__ __forceinline__ void bwd_pair(BwdPix& x, const ulonglong2 q0, const ulonglong2 q1, const float4 v0,
                                         const float4 v1, const float4 v2, float sc, float sn) {
    const u64 d[4] = {add2(q0.x, x.n[0]), add2(q0.y, x.n[1]), add2(q1.x, x.n[2]), add2(q1.y, x.n[3])};
    const float2 s = up2(fma2(d[3], d[3], fma2(d[2], d[2], fma2(d[1], d[1], mul2(d[0], d[0])))));
    const float d2 = s.x + s.y, dY = v0.x - x.Y;
    const float2 c = up2(add2(pk2(v0.z, v0.w), x.nc));
    const float c1 = c.x, c2 = c.y, cc1 = c1 * c1, cc2 = c2 * c2;
    float Ec, En;
    {  // x the centre
        const float l = ex2a(fmaf(x.kl, d2, kAdjLog2S));
        const float cw = ex2a(-fmaf(l, l, fmaf(x.K1, cc1, x.K2 * cc2)));
        const float w = sc * cw * fmaf(x.g1, c1, fmaf(x.g2, c2, x.gcd));
        Ec = l * fmaf(-w, l, sc * fmaf(x.gY, dY, x.gYd));
        x.E = fmaf(Ec, d2, x.E);
        x.c1 = fmaf(w, c1, x.c1);
        x.c2 = fmaf(w, c2, x.c2);
        x.cc1 = fmaf(w, cc1, x.cc1);
        x.cc2 = fmaf(w, cc2, x.cc2);
    }
    {  // the other pixel the centre: its differences are minus these
        const float l = ex2a(fmaf(v0.y, d2, kAdjLog2S));
        const float cw = ex2a(-fmaf(l, l, fmaf(v2.z, cc1, v2.w * cc2)));
        const float wc = sn * cw, w = wc * fmaf(-v2.x, c1, fmaf(-v2.y, c2, v1.z));
        En = l * fmaf(-w, l, sn * fmaf(-v1.x, dY, v1.y));
        x.luma = fmaf(v1.x, sn * l, x.luma);
        x.mean1 = fmaf(v2.x, wc, x.mean1);
        x.mean2 = fmaf(v2.y, wc, x.mean2);
        x.n1 = fmaf(w * v2.z, c1, x.n1);
        x.n2 = fmaf(w * v2.w, c2, x.n2);
    }
    const float G = fmaf(Ec, x.kl, En * v0.y);
    const u64 GG = pk2(G, G);
#pragma unroll
    for (int k = 0; k < 4; k++) x.p[k] = fma2(GG, d[k], x.p[k]);
}

template <int KS>
__global__ void __launch_bounds__(BwdTile<KS>::THREADS, KS == 1 ? 1 : 2) k_bm_bwd(AdjointLevelArgs a) {
    using T = BwdTile<KS>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typename T::Smem& sm = *reinterpret_cast<typename T::Smem*>(smem_raw);
    __shared__ float red[T::WARPS][6];
    const int W = a.w, H = a.h;
    const int x0 = blockIdx.x * AT_X, y0 = blockIdx.y * T::ROWS;
    const int tid = threadIdx.y * AT_X + threadIdx.x;
    const bool border = x0 < AH + 1 || y0 < AH + 1 || x0 + AT_X + AH > W - 1 || y0 + T::ROWS + AH > H - 1;
    for (int k = tid; k < T::W * T::H; k += T::THREADS) {
        const int px = x0 - AH + k % T::W, py = y0 - AH + k / T::W;
        const bool in = px >= 0 && px < W && py >= 0 && py < H;
        const size_t pi = in ? size_t(py) * W + px : 0;
        const float4* rec = reinterpret_cast<const float4*>(a.rec + pi * 12);
        const float4* pca = reinterpret_cast<const float4*>(a.pca + pi * 8);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 3; c++) sm.v[c][k] = in ? rec[c] : zero;
        sm.v[3][k] = in ? pca[0] : zero;
        sm.v[4][k] = in ? pca[1] : zero;
    }
    if (!border) {
        for (int k = tid; k < 22 * 21; k += T::THREADS) {
            const int j = k / 21, i = k % 21;
            sm.sw[j][i] = make_float2(spatial_w(i - AH, j - AH), spatial_w(i - AH, j - 1 - AH));
        }
    } else {
        // sum of the 1-D weights of the offsets d with clamp(p + d) == q
        auto weights = [&](int q, int p, int n) {
            int lo, hi;
            float v = 0.f;
            if (q >= 0 && q < n && p >= 0 && p < n && preimage(q, p, AH, n, lo, hi))
                for (int d = lo; d <= hi; d++) v += spatial_w(d, 0);
            return v;
        };
        for (int k = tid; k < (AT_X + T::ROWS) * 21; k += T::THREADS) {
            const int t = k / 21, i = k % 21;
            if (t < AT_X) {
                const int x = x0 + t, y = x + i - AH;
                sm.b.cx[t][i] = weights(y, x, W);
                sm.b.nx[t][i] = weights(x, y, W);
            } else {
                const int x = y0 + t - AT_X, y = x + i - AH;
                sm.b.y[t - AT_X][i] = make_float2(weights(y, x, H), weights(x, y, H));
            }
        }
    }
    __syncthreads();
    const int pair = threadIdx.y / KS, part = threadIdx.y % KS;
    BwdPix pix[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const int c = (2 * pair + p + AH) * T::W + threadIdx.x + AH;
        const float4 v0 = sm.v[0][c], v1 = sm.v[1][c], v2 = sm.v[2][c], p0 = sm.v[3][c], p1 = sm.v[4][c];
        BwdPix& x = pix[p];
        x.n[0] = pk2(-p0.x, -p0.y);
        x.n[1] = pk2(-p0.z, -p0.w);
        x.n[2] = pk2(-p1.x, -p1.y);
        x.n[3] = pk2(-p1.z, -p1.w);
        x.Y = v0.x;
        x.kl = v0.y;
        x.nc = pk2(-v0.z, -v0.w);
        x.gY = v1.x;
        x.gYd = v1.y;
        x.gcd = v1.z;
        x.g1 = v2.x;
        x.g2 = v2.y;
        x.K1 = v2.z;
        x.K2 = v2.w;
        x.p[0] = x.p[1] = x.p[2] = x.p[3] = 0;
        x.E = x.luma = x.c1 = x.c2 = x.cc1 = x.cc2 = x.mean1 = x.mean2 = x.n1 = x.n2 = 0.f;
    }
    const int base = 2 * pair * T::W + threadIdx.x;
    // row r of the box of the pair of pixels: row r of the upper's, r - 1 of the lower's
    auto row = [&](int r, auto up, auto lo, auto at_border) {
        float2 wu = make_float2(0.f, 0.f), wl = wu;
        if constexpr (at_border) {
            if (up) wu = sm.b.y[2 * pair][r];
            if (lo) wl = sm.b.y[2 * pair + 1][r - 1];
        }
#pragma unroll 3
        for (int i = 0; i < 21; i++) {
            const int k = base + r * T::W + i;
            const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(&sm.v[3][k]);
            const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(&sm.v[4][k]);
            const float4 v0 = sm.v[0][k], v1 = sm.v[1][k], v2 = sm.v[2][k];
            if constexpr (at_border) {
                const float c = sm.b.cx[threadIdx.x][i], n = sm.b.nx[threadIdx.x][i];
                if (up) bwd_pair(pix[0], q0, q1, v0, v1, v2, c * wu.x, n * wu.y);
                if (lo) bwd_pair(pix[1], q0, q1, v0, v1, v2, c * wl.x, n * wl.y);
            } else {
                const float2 w = sm.sw[r][i];
                if (up) bwd_pair(pix[0], q0, q1, v0, v1, v2, w.x, w.x);
                if (lo) bwd_pair(pix[1], q0, q1, v0, v1, v2, w.y, w.y);
            }
        }
    };
    auto rows = [&](auto at_border) {
        constexpr std::true_type yes{};
        constexpr std::false_type no{};
        if (part == 0) row(0, yes, no, at_border);
#pragma unroll 1
        for (int r = part == 0 ? KS : part; r <= 20; r += KS) row(r, yes, yes, at_border);
        if (part == 21 % KS) row(21, no, yes, at_border);
    };
    if (border)
        rows(std::true_type{});
    else
        rows(std::false_type{});
    if constexpr (KS > 1) {  // the parts' sums, in order
        static_assert(256 * 36 * sizeof(float) <= sizeof(typename T::Smem), "the sums take the staging's place");
        __syncthreads();
        float* t = reinterpret_cast<float*>(smem_raw) + tid;
        auto each = [&](auto f) {
#pragma unroll
            for (int p = 0; p < 2; p++) {
                BwdPix& x = pix[p];
                float* const one[10] = {&x.E, &x.luma, &x.c1, &x.c2, &x.cc1, &x.cc2, &x.mean1, &x.mean2, &x.n1, &x.n2};
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    float2 v = up2(x.p[c]);
                    f(v.x, 18 * p + 2 * c);
                    f(v.y, 18 * p + 2 * c + 1);
                    x.p[c] = pk2(v.x, v.y);
                }
#pragma unroll
                for (int c = 0; c < 10; c++) f(*one[c], 18 * p + 8 + c);
            }
        };
        each([&](float& v, int c) { t[c * 256] = v; });
        __syncthreads();
        if (part == 0) each([&](float& v, int c) {
#pragma unroll
            for (int k = 1; k < KS; k++) v += t[c * 256 + k * AT_X];
        });
    }
    float th[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int p = 0; p < 2; p++) {
        const BwdPix& v = pix[p];
        const int x = x0 + threadIdx.x, y = y0 + 2 * pair + p;
        if (part != 0 || x >= W || y >= H) continue;
        const size_t pi = size_t(y) * W + x;
        const float2 gr = *reinterpret_cast<const float2*>(a.grad + pi * 2);
        const BmScales S = bm_scales(a, v.Y, sqrtf(gr.x * gr.x + gr.y * gr.y));
        const float gL = -4.f / kAdjS * S.L * v.E;
        const float gK1 = -kAdjS * S.K1 * v.cc1, gK2 = -kAdjS * S.K2 * v.cc2;
        // scales -> centre luma and theta (ls = 1: no lens shading on this path)
        const float gsig0 = gL * S.dL_dsig0, gsig1 = gK1 * S.dK1_dsig1, gsig2 = gK2 * S.dK2_dsig2;
        const float gY = gsig0 * a.var_b[0] / (2.f * S.sig0) + gsig1 * a.var_b[1] / (2.f * S.sig1) +
                         gsig2 * a.var_b[2] / (2.f * S.sig2);
        const float aY = gsig0 / (2.f * S.sig0), aC = gsig1 / (2.f * S.sig1) + gsig2 / (2.f * S.sig2);
        th[0] += gL * (-S.L / a.tm[0]);                               // luma
        th[1] += gK1 * (-S.K1 / a.tm[1]) + gK2 * (-S.K2 / a.tm[2]);  // chroma
        th[2] += aY;                                                  // A_Y
        th[3] += aY * v.Y;                                            // B_Y
        th[4] += aC;                                                  // A_C (a[1] = a[2])
        th[5] += aC * v.Y;                                            // B_C
        *reinterpret_cast<float4*>(a.g_layer + pi * 4) =
            make_float4(gY + v.luma / kAdjS, 0.25f * kAdjS * v.mean1 + fmaf(v.K1, v.c1, v.n1) / kAdjS,
                        0.25f * kAdjS * v.mean2 + fmaf(v.K2, v.c2, v.n2) / kAdjS, 0.f);
        const float k = -4.f / (kAdjS * kAdjS * kAdjS);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const float2 u = up2(v.p[2 * c]), w = up2(v.p[2 * c + 1]);
            *reinterpret_cast<float4*>(a.g_pca + pi * 8 + 4 * c) = make_float4(k * u.x, k * u.y, k * w.x, k * w.y);
        }
    }
    // per-block theta partials, warp then block, fixed order
#pragma unroll
    for (int k = 0; k < 6; k++) {
        float v = th[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) red[tid >> 5][k] = v;
    }
    __syncthreads();
    if (tid < 6) {
        float v = 0.f;
        for (int w = 0; w < T::WARPS; w++) v += red[w][tid];
        a.part[(size_t(blockIdx.y) * gridDim.x + blockIdx.x) * 6 + tid] = v;
    }
}

// Window rows dealt to four warps while there are fewer than four 32 x 16 tiles
// for each of the chip's 148 SMs: 512x384 (384 tiles) 305 us, 339 without.
static int bwd_split(int w, int h) { return ((w + AT_X - 1) / AT_X) * ((h + 15) / 16) < 4 * 148 ? 4 : 1; }
static dim3 bwd_grid(int w, int h) {
    const int rows = bwd_split(w, h) == 4 ? BwdTile<4>::ROWS : BwdTile<1>::ROWS;
    return dim3((w + AT_X - 1) / AT_X, (h + rows - 1) / rows);
}

// pcaProjection transposed (demosaic.metal:774-796): dL/d luma(x) +=
// sum over the patches that read x of basis . dL/d pca.
// Bound by shared memory: two vertically adjacent pixels a thread read 30
// positions' 8 values (240 wavefronts a warp) and the basis (50, broadcasts)
// from a staged 36 x 20 region, 0 outside the image; 2048x1536: 131 us, 609
// with every value from global memory. Pixels on the image border, which
// several taps of a patch can read, take the general sum.
constexpr int PB_H = 16;
__global__ void __launch_bounds__(256) k_pca_bwd(AdjointLevelArgs a) {
    __shared__ float4 B[25][2], g[2][(PB_H + 4) * (AT_X + 4)];
    const int tid = threadIdx.y * AT_X + threadIdx.x;
    const int x0 = blockIdx.x * AT_X, y0 = blockIdx.y * PB_H;
    if (tid < 50) B[tid / 2][tid % 2] = reinterpret_cast<const float4*>(a.basis)[tid];
    for (int k = tid; k < 2 * (PB_H + 4) * (AT_X + 4); k += 256) {
        const int q = k >> 1, px = x0 - 2 + q % (AT_X + 4), py = y0 - 2 + q / (AT_X + 4);
        const bool in = px >= 0 && px < a.w && py >= 0 && py < a.h;
        g[k & 1][q] = in ? reinterpret_cast<const float4*>(a.g_pca)[(size_t(py) * a.w + px) * 2 + (k & 1)]
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, yt = 2 * threadIdx.y;
    float acc[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 6; r++)  // position (x + i - 2, y0 + yt + r - 2) reads x through tap 2 - i, row offset 2 - r (+ 1)
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const int q = (yt + r) * (AT_X + 4) + threadIdx.x + i;
            const float4 u = g[0][q], v = g[1][q];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const int j = 4 - r + p;
                if (j < 0 || j > 4) continue;
                const float4 b = B[j * 5 + 4 - i][0], c = B[j * 5 + 4 - i][1];
                acc[p] = fmaf(b.x, u.x, fmaf(b.y, u.y, fmaf(b.z, u.z, fmaf(b.w, u.w, acc[p]))));
                acc[p] = fmaf(c.x, v.x, fmaf(c.y, v.y, fmaf(c.z, v.z, fmaf(c.w, v.w, acc[p]))));
            }
        }
    if (x >= a.w) return;
    for (int p = 0; p < 2; p++) {
        const int y = y0 + yt + p;
        if (y >= a.h) break;
        if (x == 0 || x == a.w - 1 || y == 0 || y == a.h - 1) {
            float s = 0.f;
            for (int py = max(y - 2, 0); py <= min(y + 2, a.h - 1); py++) {
                int jlo, jhi;
                if (!preimage(y, py, 2, a.h, jlo, jhi)) continue;
                for (int px = max(x - 2, 0); px <= min(x + 2, a.w - 1); px++) {
                    int ilo, ihi;
                    if (!preimage(x, px, 2, a.w, ilo, ihi)) continue;
                    const int q = (py - y0 + 2) * (AT_X + 4) + px - x0 + 2;
                    const float4 u = g[0][q], v = g[1][q];
                    for (int j = jlo; j <= jhi; j++)
                        for (int i = ilo; i <= ihi; i++) {
                            const float4 b = B[(j + 2) * 5 + i + 2][0], c = B[(j + 2) * 5 + i + 2][1];
                            s += b.x * u.x + b.y * u.y + b.z * u.z + b.w * u.w + c.x * v.x + c.y * v.y + c.z * v.z +
                                 c.w * v.w;
                        }
                }
            }
            acc[p] = s;
        }
        a.g_layer[(size_t(y) * a.w + x) * 4] += acc[p];
    }
}

// 2 (out - target) / N through the output transform; the loss per block.
__global__ void __launch_bounds__(256) k_adj_head(const float* __restrict__ den0, const float* __restrict__ target,
                                                  int tstride, int w, int h, AdjointHeadArgs a,
                                                  float* __restrict__ g_den, double* __restrict__ loss_part) {
    __shared__ double red[8];
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (x < w && y < h) {
        const size_t pi = size_t(y) * w + x;
        const float4 d = *reinterpret_cast<const float4*>(den0 + pi * 4);
        const float v[3] = {d.x, d.y, d.z};
        float go[3];
        const float* t = target + pi * tstride;
        for (int r = 0; r < 3; r++) {
            const float o = a.m[r * 3 + 0] * v[0] + a.m[r * 3 + 1] * v[1] + a.m[r * 3 + 2] * v[2];
            const float e = o - t[r];
            l += double(e) * double(e);
            go[r] = 2.f * e * a.inv_n;
        }
        float gd[3];
        for (int c = 0; c < 3; c++) gd[c] = a.m[0 * 3 + c] * go[0] + a.m[1 * 3 + c] * go[1] + a.m[2 * 3 + c] * go[2];
        g_den[pi * 3 + 0] = gd[0];
        g_den[pi * 3 + 1] = gd[1];
        g_den[pi * 3 + 2] = gd[2];
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if ((tid & 31) == 0) red[tid >> 5] = l;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int k = 0; k < 8; k++) s += red[k];
        loss_part[size_t(blockIdx.y) * gridDim.x + blockIdx.x] = s;
    }
}

// subtractNoiseImage (demosaic.metal:922-959) transposed with respect to
// the up-sampled denoised coarse level (per fine pixel, 3 channels) and to
// the gate's noise model (nlf_a = A_Y luma, nlf_b = B_Y luma).
__global__ void __launch_bounds__(256) k_sn_bwd(AdjointSnArgs a) {
    __shared__ float red[8][2];
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    float gna = 0.f, gnb = 0.f;
    if (x < a.w && y < a.h) {
        const size_t pi = size_t(y) * a.w + x;
        const float u = (float(x) + 0.5f) * a.rx - 0.5f, v = (float(y) + 0.5f) * a.ry - 0.5f;
        const float fu = floorf(u), fv = floorf(v);
        const int xi = int(fu), yi = int(fv);
        const float ax = u - fu, ay = v - fv;
        auto bil = [&](const float* p, int c) {
            auto at = [&](int X, int Y) {
                X = clampi(X, 0, a.cw - 1);
                Y = clampi(Y, 0, a.ch - 1);
                return p[(size_t(Y) * a.cw + X) * 4 + c];
            };
            const float A = at(xi, yi), Bv = at(xi + 1, yi), Cv = at(xi, yi + 1), D = at(xi + 1, yi + 1);
            const float top = A + (Bv - A) * ax, bot = Cv + (D - Cv) * ax;
            return top + (bot - top) * ay;
        };
        const float4 ip = *reinterpret_cast<const float4*>(a.in + pi * 4);
        const float ipv[3] = {ip.x, ip.y, ip.z};
        float p1[3], pd[3], dn[3];
        for (int c = 0; c < 3; c++) {
            p1[c] = bil(a.coarse, c);
            pd[c] = bil(a.coarse_den, c);
            dn[c] = ipv[c] - (c == 0 ? a.luma_weight : 1.f) * (p1[c] - pd[c]);
        }
        float alpha = a.sharpening, dalpha_dpd0 = 0.f, dalpha_dna = 0.f, dalpha_dnb = 0.f;
        if (a.sharpening > 1.f) {
            const float2 g = *reinterpret_cast<const float2*>(a.grad + pi * 2);
            const float gm = sqrtf(g.x * g.x + g.y * g.y);
            const float sigma = sqrtf(a.nlf_a + a.nlf_b * pd[0]);
            // S1 = smoothstep(sigma, 4 sigma, gm): t = gm / (3 sigma) - 1/3
            float dS1_dt;
            const float S1 = sstep(0.f, 1.f, gm / (3.f * sigma) - 1.f / 3.f, &dS1_dt);
            const float dS1_dsig = dS1_dt * (-gm / (3.f * sigma * sigma));
            float dS2, dS3;
            const float S2 = sstep(0.75f, 0.95f, pd[0], &dS2), S3 = sstep(0.05f, 0.1f, pd[0], &dS3);
            const float detail = S1 * (1.f - S2) * S3;
            alpha = 1.f + (a.sharpening - 1.f) * detail;
            const float k = a.sharpening - 1.f;
            const float ddet_dsig = dS1_dsig * (1.f - S2) * S3;
            dalpha_dpd0 = k * (ddet_dsig * a.nlf_b / (2.f * sigma) - S1 * dS2 * S3 + S1 * (1.f - S2) * dS3);
            dalpha_dna = k * ddet_dsig / (2.f * sigma);
            dalpha_dnb = k * ddet_dsig * pd[0] / (2.f * sigma);
        }
        const float4 go4 = *reinterpret_cast<const float4*>(a.g_layer + pi * 4);
        float go[3] = {go4.x, go4.y, go4.z};
        const float o0 = pd[0] + (dn[0] - pd[0]) * alpha;
        if (!(o0 > 0.f)) go[0] = 0.f;  // max(o, 0)
        float galpha = 0.f, gpd[3];
        for (int c = 0; c < 3; c++) {
            const float wc = c == 0 ? a.luma_weight : 1.f;
            galpha += go[c] * (dn[c] - pd[c]);
            gpd[c] = go[c] * (1.f - alpha + alpha * wc);
        }
        gpd[0] += galpha * dalpha_dpd0;
        gna = galpha * dalpha_dna;
        gnb = galpha * dalpha_dnb;
        a.g_up[pi * 3 + 0] = gpd[0];
        a.g_up[pi * 3 + 1] = gpd[1];
        a.g_up[pi * 3 + 2] = gpd[2];
        if (a.g_in) {  // d(out)/d(in) = alpha, d(out)/d(up-sampled coarse) = -alpha * weight
            for (int c = 0; c < 3; c++) {
                const float wc = c == 0 ? a.luma_weight : 1.f;
                a.g_in[pi * 3 + c] += alpha * go[c];
                a.g_p1[pi * 3 + c] = -alpha * wc * go[c];
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        gna += __shfl_down_sync(0xffffffffu, gna, o);
        gnb += __shfl_down_sync(0xffffffffu, gnb, o);
    }
    if ((tid & 31) == 0) {
        red[tid >> 5][0] = gna;
        red[tid >> 5][1] = gnb;
    }
    __syncthreads();
    if (tid < 2) {
        float v = 0.f;
        for (int w = 0; w < 8; w++) v += red[w][tid];
        a.part[(size_t(blockIdx.y) * gridDim.x + blockIdx.x) * 2 + tid] = v;
    }
}

// bilinear up-sampling (the reconstruct step's coarse reads) transposed:
// each coarse pixel gathers the weights with which fine pixels sampled it.
__device__ __forceinline__ void up_transpose(const AdjointSnArgs& a, const float* src, float* dst, bool accumulate) {
    const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y * blockDim.y + threadIdx.y;
    if (X >= a.cw || Y >= a.ch) return;
    float acc[3] = {0, 0, 0};
    for (int y = max(2 * Y - 4, 0); y <= min(2 * Y + 4, a.h - 1); y++) {
        const float v = (float(y) + 0.5f) * a.ry - 0.5f;
        const float fv = floorf(v);
        const int yi = int(fv);
        const float ay = v - fv;
        const float wy = (clampi(yi, 0, a.ch - 1) == Y ? 1.f - ay : 0.f) + (clampi(yi + 1, 0, a.ch - 1) == Y ? ay : 0.f);
        if (wy == 0.f) continue;
        for (int x = max(2 * X - 4, 0); x <= min(2 * X + 4, a.w - 1); x++) {
            const float u = (float(x) + 0.5f) * a.rx - 0.5f;
            const float fu = floorf(u);
            const int xi = int(fu);
            const float ax = u - fu;
            const float wx =
                (clampi(xi, 0, a.cw - 1) == X ? 1.f - ax : 0.f) + (clampi(xi + 1, 0, a.cw - 1) == X ? ax : 0.f);
            if (wx == 0.f) continue;
            const float* g = src + (size_t(y) * a.w + x) * 3;
            const float wgt = wx * wy;
            acc[0] += wgt * g[0];
            acc[1] += wgt * g[1];
            acc[2] += wgt * g[2];
        }
    }
    float* o = dst + (size_t(Y) * a.cw + X) * 3;
    for (int c = 0; c < 3; c++) o[c] = accumulate ? o[c] + acc[c] : acc[c];
}

__global__ void __launch_bounds__(256) k_up_bwd(AdjointSnArgs a) { up_transpose(a, a.g_up, a.g_coarse_den, false); }
__global__ void __launch_bounds__(256) k_up_bwd_img(AdjointSnArgs a) { up_transpose(a, a.g_p1, a.g_coarse_img, true); }

// k_downsample transposed: out(x, y) = 1/4 sum over a, b in {0, 1} of the
// bilinear sample at (x rx - 0.5 + a rx, y ry - 0.5 + b ry), clamp-to-edge,
// a separable weight; each fine pixel gathers from the coarse pixels whose
// samples touch it.
__device__ __forceinline__ float down_weight(int X, int x, float r, int n) {
    float wsum = 0.f;
    for (int t = 0; t < 2; t++) {
        const float u = __fsub_rn(__fmul_rn(float(x + t), r), 0.5f);
        const float fu = floorf(u);
        const int xi = int(fu);
        const float ax = u - fu;
        wsum += (clampi(xi, 0, n - 1) == X ? 1.f - ax : 0.f) + (clampi(xi + 1, 0, n - 1) == X ? ax : 0.f);
    }
    return wsum;
}

__global__ void __launch_bounds__(256) k_down_bwd(const float* __restrict__ gc, int cw, int ch, float* __restrict__ gf,
                                                 int w, int h, float rx, float ry) {
    const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y * blockDim.y + threadIdx.y;
    if (X >= w || Y >= h) return;
    const int x0 = max(int(floorf(float(X) / rx)) - 3, 0), x1 = min(int(floorf(float(X) / rx)) + 3, cw - 1);
    const int y0 = max(int(floorf(float(Y) / ry)) - 3, 0), y1 = min(int(floorf(float(Y) / ry)) + 3, ch - 1);
    float acc[3] = {0, 0, 0};
    for (int y = y0; y <= y1; y++) {
        const float wy = down_weight(Y, y, ry, h);
        if (wy == 0.f) continue;
        for (int x = x0; x <= x1; x++) {
            const float wx = down_weight(X, x, rx, w);
            if (wx == 0.f) continue;
            const float wgt = 0.25f * wx * wy;
            const float* g = gc + (size_t(y) * cw + x) * 3;
            acc[0] += wgt * g[0];
            acc[1] += wgt * g[1];
            acc[2] += wgt * g[2];
        }
    }
    float* o = gf + (size_t(Y) * w + X) * 3;
    o[0] += acc[0];
    o[1] += acc[1];
    o[2] += acc[2];
}

__global__ void __launch_bounds__(256) k_add_layer_grad(const float* __restrict__ gl, float* __restrict__ gi, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int c = 0; c < 3; c++) gi[size_t(i) * 3 + c] += gl[size_t(i) * 4 + c];
}

// 3-channel gradient planes to and from caller views of 3 or 4 channels
__global__ void __launch_bounds__(256) k_pack3(const float* __restrict__ src, size_t pitch, int ch,
                                              float* __restrict__ dst, int w, int h) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float* p = src + size_t(y) * pitch + size_t(x) * ch;
    float* o = dst + (size_t(y) * w + x) * 3;
    o[0] = p[0];
    o[1] = p[1];
    o[2] = p[2];
}

__global__ void __launch_bounds__(256) k_unpack3(const float* __restrict__ src, float* __restrict__ dst, size_t pitch,
                                                int ch, int w, int h) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const float* p = src + (size_t(y) * w + x) * 3;
    float* o = dst + size_t(y) * pitch + size_t(x) * ch;
    o[0] = p[0];
    o[1] = p[1];
    o[2] = p[2];
    if (ch == 4) o[3] = 0.f;
}

void launch_pack3(const float* src, size_t pitch_floats, int channels, float* dst, int w, int h, cudaStream_t s) {
    const dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    k_pack3<<<g, b, 0, s>>>(src, pitch_floats, channels, dst, w, h);
}

void launch_unpack3(const float* src, float* dst, size_t pitch_floats, int channels, int w, int h, cudaStream_t s) {
    const dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    k_unpack3<<<g, b, 0, s>>>(src, dst, pitch_floats, channels, w, h);
}

void launch_adj_head(const float* den0, const float* target, int tstride, int w, int h, const AdjointHeadArgs& a,
                     float* g_den, double* loss_part, cudaStream_t s) {
    const dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    k_adj_head<<<g, b, 0, s>>>(den0, target, tstride, w, h, a, g_den, loss_part);
}

void launch_bm_bwd(const AdjointLevelArgs& a, cudaStream_t s) {
    const dim3 b2(32, 8), g2((a.w + 31) / 32, (a.h + 7) / 8), g = bwd_grid(a.w, a.h);
    k_bm_bwd_record<<<g2, b2, 0, s>>>(a);
    auto run = [&](auto kernel, int warps, size_t bytes) {
        ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), int(bytes));
        kernel<<<g, dim3(AT_X, warps), bytes, s>>>(a);
    };
    if (bwd_split(a.w, a.h) == 4)
        run(k_bm_bwd<4>, BwdTile<4>::WARPS, sizeof(BwdTile<4>::Smem));
    else
        run(k_bm_bwd<1>, BwdTile<1>::WARPS, sizeof(BwdTile<1>::Smem));
    k_pca_bwd<<<dim3((a.w + AT_X - 1) / AT_X, (a.h + PB_H - 1) / PB_H), dim3(AT_X, PB_H / 2), 0, s>>>(a);
}

void launch_sn_bwd(const AdjointSnArgs& a, cudaStream_t s) {
    const dim3 b(32, 8), g((a.w + 31) / 32, (a.h + 7) / 8), gc((a.cw + 31) / 32, (a.ch + 7) / 8);
    k_sn_bwd<<<g, b, 0, s>>>(a);
    k_up_bwd<<<gc, b, 0, s>>>(a);
    if (a.g_in) k_up_bwd_img<<<gc, b, 0, s>>>(a);
}

void launch_add_layer_grad(const float* g_layer, float* g_img, int w, int h, cudaStream_t s) {
    const int n = w * h;
    k_add_layer_grad<<<(n + 255) / 256, 256, 0, s>>>(g_layer, g_img, n);
}

void launch_down_bwd(const float* g_coarse, int cw, int ch, float* g_fine, int w, int h, cudaStream_t s) {
    const dim3 b(32, 8), g((w + 31) / 32, (h + 7) / 8);
    k_down_bwd<<<g, b, 0, s>>>(g_coarse, cw, ch, g_fine, w, h, float(w) / float(cw), float(h) / float(ch));
}

int adjoint_blocks(int w, int h) {
    const dim3 g = bwd_grid(w, h);
    return int(g.x * g.y);
}
int adjoint_sn_blocks(int w, int h) { return ((w + 31) / 32) * ((h + 7) / 8); }

}  // namespace gls
