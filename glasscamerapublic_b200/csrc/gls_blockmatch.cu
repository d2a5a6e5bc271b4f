// gls_blockmatch.cu — blockMatchingDenoiseImage (demosaic.metal:806-884):
// 21 x 21 non-local means with a PCA-space patch distance for luma, a
// chroma distance for chroma and a fixed spatial Gaussian:
//   lw = exp(-2 (|p - q|_8 s)^2),   s = 1 / (luma_mult sigma_Y (1 + gb edge))
//   cw = exp(-2 (lw^2 + (dCb m1 / cb)^2 + (dCr m2 / cb)^2))
//   w  = gaussian(0.1 |(i, j)|) * (lw, cw, cw)
// accumulated in FP32; output (Y, Cb, Cr, sum of luma weights).
//
// The kernels stage the tile's window region (halo 10) in shared memory. The
// one for the FP32 plain path evaluates the formula directly, two vertically
// adjacent pixels a thread; the FP16-storage path's forms the distances on the
// tensor cores and the weights and sums in packed FP32.
#include <cmath>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <shared_mutex>

#include "gls_common.cuh"
#include "gls_kernels.h"
#include "gls_pyramid_dev.cuh"

namespace gls {

__device__ __forceinline__ __half2 u2h_(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Per-pixel constants of the matchers.
struct BmConst {
    float s;       // luma distance scale
    float c1, c2;  // chroma scales (dm / chroma_boost)
};

template <class S>
__device__ __forceinline__ BmConst bm_const(const BlockMatchArgs& a, Plane<S, 2> grad, int w, int h, int px, int py,
                                            float y) {
    BmConst k;
    float ls = 1.f;
    if (a.lsc > 0.f) {  // lensShading, demosaic.metal:91-93, at the pixel
        const float cx = float(w / 2), cy = float(h / 2);
        const float dx = float(px) - cx, dy = float(py) - cy;
        const float rr = sqrtf(dx * dx + dy * dy) / sqrtf(cx * cx + cy * cy);
        ls = 1.f + a.lsc * rr * rr;
    }
    const float sig0 = sqrtf(a.var_a[0] + a.var_b[0] * ls * y);
    const float sig1 = sqrtf(a.var_a[1] + a.var_b[1] * ls * y);
    const float sig2 = sqrtf(a.var_a[2] + a.var_b[2] * ls * y);
    const float dm0 = 1.f / (a.tm[0] * sig0), dm1 = 1.f / (a.tm[1] * sig1), dm2 = 1.f / (a.tm[2] * sig2);
    const f2 g = ld2<S>(grad.px(px, py));
    const float mag = sqrtf(g.x * g.x + g.y * g.y);
    const float edge = smoothstepf(2.f, 16.f, a.gradient_threshold * mag / sig0);
    k.s = dm0 / (1.f + a.gradient_boost * edge);
    k.c1 = dm1 / a.chroma_boost;
    k.c2 = dm2 / a.chroma_boost;
    return k;
}

__device__ __forceinline__ float spatial_weight(int i, int j) {  // gaussian(0.1 |(i, j)|)
    const float d = 0.1f * sqrtf(float(i * i + j * j));
    return expf(-2.f * d * d);
}

typedef unsigned long long u64;

__device__ __forceinline__ u64 pk2(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(u64 r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
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

// ============================================================ FP32 plain path
// NP vertically adjacent pixels per thread, 32 x 4 threads, FP32 staging. The
// arithmetic of a tap and the order of a window's sums (row by row) are the
// same whatever the tile, so every tile gives the same bits. Differences and
// chroma terms are packed FP32 (the same roundings in half the instructions),
// the distance's sum stays a serial chain; ex2.approx.ftz where exp2f only
// adds the scaling that keeps results below 2^-126, which count for the pixels
// of bmp_chroma_again alone.
//
// What bounds it: two pixels' tap takes 60 cycles of a sub-partition's FMA
// pipe, 32 of its MUFU and 57 issue slots, and the SM's shared memory serves
// four of them in 52 wavefronts. The coefficients lie in two arrays because a
// warp's 16-byte loads at a 32-byte stride hit each bank twice (84 wavefronts,
// the former bound). 1024x768: 550 -> 428 us, 128x96: 63 -> 23 us; three
// blocks of 32 x 8 pixels an SM where two of 32 x 16 leave a longer last wave
// (512x384: 125 us with those).
template <int NP>
struct BmPlainTile {
    static constexpr int TX = 32, TY = 4, THREADS = TX * TY, ROWS = NP * TY;
    static constexpr int W = TX + 20, H = ROWS + 20;
    struct Smem {
        ulonglong2 pca0[H * W], pca1[H * W];  // coefficients 0..3, 4..7
        float4 ycc[H * W];                    // Cb, Cr, Y
        float2 spatial[22][21];               // the weights of window rows j and j - 1
    };
};

struct BmPlainPix {
    u64 n[4];   // minus the coefficients
    float kl;   // -2 log2(e) s^2
    u64 c, no;  // sqrt(2 log2 e) (c1, c2), minus that times the centre chroma
};

// One row of the union of the pixels' windows: the upper pixel's taps when UP,
// the lower's when LO.
template <bool UP, bool LO, int NP, class Smem>
__device__ __forceinline__ void bmp_row(const Smem& sm, int base, int r, const BmPlainPix (&pix)[NP],
                                        float (&acc)[NP][5]) {
    const float kLk = 2.f * 1.4426950408889634f;
#pragma unroll
    for (int i = 0; i < 21; i++) {
        const ulonglong2 q0 = sm.pca0[base + i], q1 = sm.pca1[base + i];
        const float4 y = sm.ycc[base + i];
        const float2 sw = sm.spatial[r][i];
        const u64 ch = pk2(y.x, y.y);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            if (p == 0 ? !UP : !LO) continue;
            const BmPlainPix& P = pix[p];
            float(&s)[5] = acc[p];
            float d[8], e1, e2;
            upk2(add2(q0.x, P.n[0]), d[0], d[1]);
            upk2(add2(q0.y, P.n[1]), d[2], d[3]);
            upk2(add2(q1.x, P.n[2]), d[4], d[5]);
            upk2(add2(q1.y, P.n[3]), d[6], d[7]);
            float d2 = d[0] * d[0];
#pragma unroll
            for (int k = 1; k < 8; k++) d2 = fmaf(d[k], d[k], d2);
            const float lw = ex2_approx(P.kl * d2);
            upk2(fma2(P.c, ch, P.no), e1, e2);
            const float cw = ex2_approx(-fmaf(kLk * lw, lw, fmaf(e1, e1, e2 * e2)));
            const float w = p == 0 ? sw.x : sw.y;
            const float wy = w * lw, wc = w * cw;
            s[0] = fmaf(wy, y.z, s[0]);
            s[1] = fmaf(wc, y.x, s[1]);
            s[2] = fmaf(wc, y.y, s[2]);
            s[3] += wy;
            s[4] += wc;
        }
    }
}

// A pixel whose chroma weights are all so small that those below 2^-126, which
// ex2.approx.ftz drops, count (scales at which the rounding of c times the pixel's
// own chroma alone reaches the exponent's range): the chroma sums once more by
// exp2f, which keeps them down to 2^-149.
template <class Smem>
__device__ __forceinline__ void bmp_chroma_again(const Smem& sm, int base, int pitch, const BmPlainPix& P,
                                              float (&s)[5]) {
    const float kLk = 2.f * 1.4426950408889634f;
    s[1] = s[2] = s[4] = 0.f;
#pragma unroll 1
    for (int k = 0; k < 441; k++) {
        const int j = k / 21, i = k % 21, q = base + j * pitch + i;
        const ulonglong2 q0 = sm.pca0[q], q1 = sm.pca1[q];
        const float4 y = sm.ycc[q];
        float d[8], e1, e2;
        upk2(add2(q0.x, P.n[0]), d[0], d[1]);
        upk2(add2(q0.y, P.n[1]), d[2], d[3]);
        upk2(add2(q1.x, P.n[2]), d[4], d[5]);
        upk2(add2(q1.y, P.n[3]), d[6], d[7]);
        float d2 = d[0] * d[0];
        for (int c = 1; c < 8; c++) d2 = fmaf(d[c], d[c], d2);
        const float lw = exp2f(P.kl * d2);
        upk2(fma2(P.c, pk2(y.x, y.y), P.no), e1, e2);
        const float wc = sm.spatial[j][i].x * exp2f(-fmaf(kLk * lw, lw, fmaf(e1, e1, e2 * e2)));
        s[1] = fmaf(wc, y.x, s[1]);
        s[2] = fmaf(wc, y.y, s[2]);
        s[4] += wc;
    }
}

template <int NP>
__global__ void __launch_bounds__(128, 3)
    k_block_match_plain(Plane<float, 4> img, Plane<float, 2> grad, Plane<float, 8> pca, Plane<float, 4> out,
                        BlockMatchArgs a) {
    using T = BmPlainTile<NP>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typename T::Smem& sm = *reinterpret_cast<typename T::Smem*>(smem_raw);
    const int x0 = blockIdx.x * T::TX, y0 = blockIdx.y * T::ROWS;
    const int tid = threadIdx.y * T::TX + threadIdx.x;
    for (int k = tid; k < 22 * 21; k += T::THREADS) {
        const int j = k / 21, i = k % 21;
        sm.spatial[j][i] = make_float2(spatial_weight(i - 10, j - 10), spatial_weight(i - 10, j - 11));
    }
    for (int k = tid; k < T::W * T::H; k += T::THREADS) {
        const int ty = k / T::W, tx = k % T::W;
        const int sx = clampi(x0 - 10 + tx, 0, img.w - 1), sy = clampi(y0 - 10 + ty, 0, img.h - 1);
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(pca.px(sx, sy));
        sm.pca0[k] = q[0];
        sm.pca1[k] = q[1];
        const f4 p = ld4<float>(img.px(sx, sy));
        sm.ycc[k] = make_float4(p.y, p.z, p.x, 0.f);
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, y = y0 + NP * threadIdx.y;
    const float kLog2e = 1.4426950408889634f, sq = sqrtf(2.f * kLog2e);
    BmPlainPix pix[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int c = (NP * threadIdx.y + p + 10) * T::W + threadIdx.x + 10;
        const float4 in = sm.ycc[c];
        const BmConst k = bm_const<float>(a, grad, img.w, img.h, min(x, img.w - 1), min(y + p, img.h - 1), in.z);
        BmPlainPix& P = pix[p];
        const float4 p0 = *reinterpret_cast<const float4*>(&sm.pca0[c]), p1 = *reinterpret_cast<const float4*>(&sm.pca1[c]);
        P.n[0] = pk2(-p0.x, -p0.y);
        P.n[1] = pk2(-p0.z, -p0.w);
        P.n[2] = pk2(-p1.x, -p1.y);
        P.n[3] = pk2(-p1.z, -p1.w);
        P.kl = -2.f * kLog2e * k.s * k.s;
        const float c1 = sq * k.c1, c2 = sq * k.c2;
        P.c = pk2(c1, c2);
        P.no = pk2(-(c1 * in.x), -(c2 * in.y));
    }
    float acc[NP][5] = {};
    const int base = NP * threadIdx.y * T::W + threadIdx.x;
    if constexpr (NP == 2) {
        bmp_row<true, false, NP>(sm, base, 0, pix, acc);
#pragma unroll 1
        for (int r = 1; r <= 20; r++) bmp_row<true, true, NP>(sm, base + r * T::W, r, pix, acc);
        bmp_row<false, true, NP>(sm, base + 21 * T::W, 21, pix, acc);
    } else {
#pragma unroll 1
        for (int r = 0; r <= 20; r++) bmp_row<true, false, NP>(sm, base + r * T::W, r, pix, acc);
    }
    if (x >= out.w) return;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        if (y + p >= out.h) continue;
        float(&s)[5] = acc[p];
        if (s[4] < 0x1p-80f) bmp_chroma_again(sm, base + p * T::W, T::W, pix[p], s);
        st4<float>(out.px(x, y + p), f4{s[0] / s[3], s[1] / s[4], s[2] / s[4], s[3]});
        if (a.nc_out) a.nc_out[size_t(y + p) * out.w + x] = s[4];
    }
}

// ============================================================ FP16-storage path
// Distances on the tensor cores, weights and sums in packed FP32. A warp takes
// a group of 4 x 2 pixels: the union of their windows is 24 x 22 positions, of
// which each pixel's 21 x 21 window is 83.5%, walked as 33 tiles of 16
// neighbours (2 rows x 8 columns). Per tile
//   * S = |q'|^2 / 2 - p'.q' for 16 neighbours x 8 pixels by one mma.sync
//     m16n8k8: A holds the neighbours' centred coefficients (8 halves), B the
//     pixels' negated (any finite half stays one; twice them need not), C the
//     neighbours' |q'|^2 / 2 in FP32. Products of
//     halves are exact in FP32; the MMA's sum of nine terms does not round each
//     addition to nearest, but rounds fewer times than a chain of FP32 FMAs: the
//     exponents' error against float64 is 0.8 to 0.96 of the chain's (rms; the largest
//     0.6 to 1.0 of it) for coefficients of 0 to 300 times their noise; centring on
//     the tile-centre pixel's coefficients keeps the cancellation error at FP32
//     rounding of the local variation of the coefficients;
//   * a lane gets S of two horizontally adjacent pixels for each of two
//     neighbours and evaluates both pixels' weights as packed FP32 pairs
//     (fma/mul/add .rn.f32x2), the neighbour's values staged twice so that one
//     load gives the broadcast pair: lw scaled by sqrt(2 log2 e) =
//     exp2(2 kl S + base), chroma weight exp2(-(lw^2 + d1^2 + d2^2 - log2 sw)),
//     both by ex2.approx.f32 (the reference uses half-precision exp under fast
//     math here), then the five FP32 sums;
//   * the spatial weight is separable. Its row part comes from a 23-entry table
//     (weight 0, log-weight -inf outside the window's rows); its column part is
//     fixed for a lane and column segment, so the sums are kept per segment
//     and multiplied by it once at the end (0 outside the window's columns).
// The lanes' sums are added over the 8 neighbour columns at the end.
//
// What bounds it: per tile and warp 8 ex2 (64 cycles of the sub-partition's
// MUFU), 24 packed FP32 instructions (56 cycles of its FMA pipe) and about 46
// issue slots, so the MUFU's 3.69 ms per 12 MP frame (5 levels) is the floor.
// Measured: level 0 of a 2016x1512 image 1.24 ms (1.64 ms with the scalar
// distance in packed FP32, four pixels a thread), 83 cycles a tile in the loop
// (the mix of 8 ex2 and 24 packed FMA alone runs at about 70) and a quarter of
// the time in staging, projection and the groups' ends; XU pipe 64% busy, issue
// slots 60%. The five levels of a 12 MP frame: 7.23 -> 6.41 ms.
constexpr int BX_TX = 32, BX_W = BX_TX + 20;
// tile variants: TY warps of 32 NP pixels, tiles of 32 x (NP TY) = 32 x 32 or
// 32 x 16 pixels (bm_tile_variant chooses).
// Variant code 10 TY + NP: 84, 44, 82, 162. A 32 x 32 tile's staging takes an
// SM's shared memory alone, a 32 x 16 tile's half of it.
template <int TY, int NP>
struct BxTile {
    static constexpr int ROWS = NP * TY;
    static constexpr int H = ROWS + 20;     // window rows staged
    static constexpr int LH = H + 4;        // luma rows staged
    static constexpr int THREADS = BX_TX * TY;
    static constexpr int MIN_BLOCKS = ROWS == 16 ? 2 : 1;
    static_assert(ROWS == 16 || ROWS == 32, "tile heights divide the 32-row centring tiles");
    static_assert((BX_W * H) % 16 == 0, "the projection takes 16 positions at a time");
};
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ uint32_t hmul2_u(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void mma1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, float c0, float c1,
                                        float c2, float c3) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

constexpr int BX_LW = BX_W + 4;  // luma tile width, origin (x0 - 12, y0 - 12)

enum { BK_KL, BK_BASE, BK_C1, BK_C2, BK_NO1, BK_NO2, BK_COUNT };

// shared memory of a tile
template <int TY, int NP>
struct BmTileSmem {
    using T = BxTile<TY, NP>;
    uint4 q[T::H * BX_W];                  // q - c, 8 halves
    float4 yb[T::H * BX_W];                // (Y, Y, Cb, Cb)
    float2 cr[T::H * BX_W];                // (Cr, Cr)
    float2 nn[T::H * BX_W];                // (|q - c|^2 / 2, the same)
    float4 wrow[24];                       // row part of the spatial weight, dy = -11 .. 11: (-log2, -log2, w / sqrt(lk) twice)
    float wcol[28];                        // column part, dx = -13 .. 13
    float cen[8];
    float bsm[25][8];
    float k[BK_COUNT][T::ROWS * BX_TX];    // per pixel: 2 kl, base, c1, c2, -c1 Cb, -c2 Cr
    __half luma[2][T::LH * BX_LW];         // the luma tile, and the same shifted left by one
    unsigned nn_max, kl_max;               // bits of the largest |q - c|^2 / 2 and |2 kl|
};

// a lane's view of a group: two adjacent pixels' constants as pairs
struct BmPair {
    u64 kl, base, c1, c2, no1, no2;
};

// The weights of a pixel pair for one neighbour and the five sums. S: the
// pair's distances; yy, cb, cr: the neighbour's values; ly, sy: the row part of
// the spatial weight, -log2 and over sqrt(lk).
template <bool CLAMP>
__device__ __forceinline__ void bm_accumulate(const BmPair& P, u64 S, u64 yy, u64 cb, u64 cr, u64 ly, u64 sy,
                                              u64 (&acc)[5]) {
    float e0, e1, l0, l1, n0, n1;
    upk2(fma2(P.kl, S, P.base), e0, e1);
    // the exponent is at most log2 sqrt(lk) but for rounding, held below 2
    l0 = ex2_approx(CLAMP ? fminf(e0, 2.f) : e0);
    l1 = ex2_approx(CLAMP ? fminf(e1, 2.f) : e1);
    const u64 lws = pk2(l0, l1);
    const u64 d1 = fma2(P.c1, cb, P.no1), d2 = fma2(P.c2, cr, P.no2);
    upk2(fma2(lws, lws, fma2(d1, d1, fma2(d2, d2, ly))), n0, n1);
    const u64 wc = pk2(ex2_approx(-n0), ex2_approx(-n1));
    const u64 wy = mul2(sy, lws);
    acc[0] = fma2(wy, yy, acc[0]);
    acc[1] = fma2(wc, cb, acc[1]);
    acc[2] = fma2(wc, cr, acc[2]);
    acc[3] = add2(acc[3], wy);
    acc[4] = add2(acc[4], wc);
}

__device__ __forceinline__ u64 as_u64(float2 v) { return pk2(v.x, v.y); }

// The sums of one group (pixel origin gx, gy in the tile). SAFE: positions
// outside a pixel's window are read as 0, so that a value that is not finite
// reaches the pixels whose windows hold it (a luma: a patch that holds it, so
// up to 12 positions away) and no others. CLAMP: the luma
// exponents may round past their limit.
template <bool SAFE, bool CLAMP, class Sm>
__device__ __forceinline__ void bm_group(const Sm& sm, int gx, int gy, u64 (&acc)[3][5]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    BmPair P;
    {
        const int i = (gy + (t >> 1)) * BX_TX + gx + 2 * (t & 1);
        auto pair = [&](int c) { return as_u64(*reinterpret_cast<const float2*>(&sm.k[c][i])); };
        P = {pair(BK_KL), pair(BK_BASE), pair(BK_C1), pair(BK_C2), pair(BK_NO1), pair(BK_NO2)};
    }
    // B: minus pixel g's coefficients 2t, 2t + 1
    const uint32_t* q32 = reinterpret_cast<const uint32_t*>(sm.q);
    const uint32_t bq = q32[((gy + (g >> 2) + 10) * BX_W + gx + (g & 3) + 10) * 4 + t] ^ 0x80008000u;
#pragma unroll
    for (int k = 0; k < 15; k++) acc[k / 5][k % 5] = 0;
    // neighbour g of a tile's first row; ldmatrix: lanes 0-7 the first row's
    // eight positions, lanes 8-15 the second row's
    int pos = gy * BX_W + gx + g;
    uint32_t lda = uint32_t(__cvta_generic_to_shared(&sm.q[(gy + ((lane >> 3) & 1)) * BX_W + gx + (lane & 7)]));
    const float4* wr = &sm.wrow[1 - (t >> 1)];
#pragma unroll 1
    for (int r = 0; r < 11; r++, pos += 2 * BX_W, lda += 2 * BX_W * 16, wr += 2) {
        const float4 w0 = wr[0], w1 = wr[1];
#pragma unroll
        for (int s = 0; s < 3; s++) {
            uint32_t a0, a1;
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];"
                         : "=r"(a0), "=r"(a1)
                         : "r"(lda + 8 * 16 * s));
            const int p0 = pos + 8 * s, p1 = p0 + BX_W;
            const float2 m0 = sm.nn[p0], m1 = sm.nn[p1];
            float S[4];
            mma1688(S, a0, a1, bq, m0.x, m0.y, m1.x, m1.y);
            float4 y0 = sm.yb[p0], y1 = sm.yb[p1];
            float2 c0 = sm.cr[p0], c1 = sm.cr[p1];
            if constexpr (SAFE) {
                const int dx = 8 * s + g - 2 * (t & 1) - 10, dy = 2 * r - (t >> 1) - 10;
                auto zero = [&](float4& y, float2& c, float& s0, float& s1, int d) {
                    const bool row = d >= -10 && d <= 10, in0 = row && dx >= -10 && dx <= 10,
                               in1 = row && dx - 1 >= -10 && dx - 1 <= 10;
                    y.x = in0 ? y.x : 0.f, y.z = in0 ? y.z : 0.f, c.x = in0 ? c.x : 0.f, s0 = in0 ? s0 : 0.f;
                    y.y = in1 ? y.y : 0.f, y.w = in1 ? y.w : 0.f, c.y = in1 ? c.y : 0.f, s1 = in1 ? s1 : 0.f;
                };
                zero(y0, c0, S[0], S[1], dy);
                zero(y1, c1, S[2], S[3], dy + 1);
            }
            bm_accumulate<CLAMP>(P, pk2(S[0], S[1]), pk2(y0.x, y0.y), pk2(y0.z, y0.w), as_u64(c0),
                                 pk2(w0.x, w0.y), pk2(w0.z, w0.w), acc[s]);
            bm_accumulate<CLAMP>(P, pk2(S[2], S[3]), pk2(y1.x, y1.y), pk2(y1.z, y1.w), as_u64(c1),
                                 pk2(w1.x, w1.y), pk2(w1.z, w1.w), acc[s]);
        }
    }
}

// A warp's share of the tile's groups (of the part `part` of `parts`), the
// results into shared memory.
template <bool SAFE, bool CLAMP, int TY, class Sm>
__device__ __forceinline__ void bm_groups(Sm& sm, int part, int parts) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    constexpr int GROUPS = (BX_TX / 4) * (Sm::T::ROWS / 2);
    // the column part of the spatial weight: neighbour g of each segment,
    // pixel columns 2 (t & 1) and 2 (t & 1) + 1
    u64 sx[3];
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const float* w = &sm.wcol[8 * s + g - 2 * (t & 1) - 10 + 13];
        sx[s] = pk2(w[0], w[-1]);
    }
    const bool second = lane & 16;
#pragma unroll 1
    for (int grp = warp + TY * part; grp < GROUPS; grp += TY * parts) {
        const int gx = (grp % (BX_TX / 4)) * 4, gy = (grp / (BX_TX / 4)) * 2;
        u64 part[3][5];
        bm_group<SAFE, CLAMP>(sm, gx, gy, part);
        // over the eight neighbour columns: lanes of the lower half keep the
        // first pixel of their pair, those of the upper half the second
        float v[5];
#pragma unroll
        for (int k = 0; k < 5; k++) {
            float u0, u1;
            upk2(fma2(sx[2], part[2][k], fma2(sx[1], part[1][k], mul2(sx[0], part[0][k]))), u0, u1);
            v[k] = (second ? u1 : u0) + __shfl_xor_sync(0xffffffffu, second ? u0 : u1, 16);
        }
#pragma unroll
        for (int k = 0; k < 5; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], 8);
#pragma unroll
        for (int k = 0; k < 5; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], 4);
        // into the place of the pixel's constants, which only this group reads
        if ((lane & 12) == 0) {
            const int i = (gy + (t >> 1)) * BX_TX + gx + 2 * (t & 1) + second;
#pragma unroll
            for (int k = 0; k < 5; k++) sm.k[k][i] = v[k];
        }
    }
}

// One tile (origin x0, y0) by TY warps. Shared by the stream kernel and the
// persistent kernel's block-matching tasks.
template <int TY, int NP>
__device__ __forceinline__ void bm_tile(int x0, int y0, const Plane<__half, 4>& img, const Plane<__half, 2>& grad,
                                        const float* __restrict__ basis, const Plane<__half, 4>& out,
                                        const BlockMatchArgs& a, BmTileSmem<TY, NP>& sm, int part = 0, int parts = 1) {
    using T = BxTile<TY, NP>;
    constexpr int NT = T::THREADS, NPOS = BX_W * T::H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const float kLog2e = 1.4426950408889634f, lk = 2.f * kLog2e, isq = rsqrtf(lk);
    const float inf = __int_as_float(0x7f800000);
    if (tid < 27) {
        const int d = tid - 13;
        sm.wcol[tid] = d >= -10 && d <= 10 ? spatial_weight(d, 0) : 0.f;
    } else if (tid >= 32 && tid < 32 + 23) {
        const int d = tid - 32 - 11;
        const float w = d >= -10 && d <= 10 ? spatial_weight(0, d) : 0.f, l = w > 0.f ? -log2f(w) : inf;
        sm.wrow[tid - 32] = make_float4(l, l, w * isq, w * isq);
    }
    for (int k = tid; k < 200; k += NT) sm.bsm[k / 8][k % 8] = basis[k];
    if (tid == 0) sm.nn_max = sm.kl_max = 0;
    // the window region plus the patches' margin of 2, a warp per row
    bool bad = false;  // a staged value that is not finite
#pragma unroll
    for (int i = 0; i < (T::LH + TY - 1) / TY; i++) {  // unrolled: all of a warp's loads in flight
        const int ty = warp + i * TY;
        if (ty >= T::LH) break;
        const __half* row = img.px(0, clampi(y0 - 12 + ty, 0, img.h - 1));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int tx = lane + 32 * h;
            if (tx >= BX_LW) break;
            const __half* src = row + 4 * clampi(x0 - 12 + tx, 0, img.w - 1);
            const __half y = *src;
            const f4 p = ld4<__half>(src);
            const int l = ty * BX_LW + tx, k = (ty - 2) * BX_W + tx - 2;
            sm.luma[0][l] = y;
            if (tx > 0) sm.luma[1][l - 1] = y;
            bad = bad || !(fabsf(p.x) + fabsf(p.y) + fabsf(p.z) < inf);
            if (ty >= 2 && ty < T::H + 2 && tx >= 2 && tx < BX_W + 2) {
                sm.yb[k] = make_float4(p.x, p.x, p.y, p.y);
                sm.cr[k] = make_float2(p.z, p.z);
            }
        }
    }
    __syncthreads();
    if (tid < 8) {  // centring vector: the coefficients (FP32) of the centre pixel of the
                    // enclosing 32 x 32 tile, so that both tile heights centre and round alike
        const int cx = BX_TX / 2 + 12, cy = 16 + 12 - (y0 % 32);  // luma-tile coordinates
        // (any finite centre will do: a luma that is not finite is taken as the one before it,
        // so that it spoils the positions whose patches hold it and not the whole tile)
        float c = 0.f, y = 0.f;
        for (int k = 0; k < 25; k++) {
            const float v = __half2float(sm.luma[0][(cy + k / 5 - 2) * BX_LW + cx + k % 5 - 2]);
            y = fabsf(v) < inf ? v : y;
            c += sm.bsm[k][tid] * y;
        }
        sm.cen[tid] = c;
    }
    // pcaProjection (demosaic.metal:774-796) fused into the tile producer: the
    // 5x5 luma patch of every window position times the 25 x 8 basis, as FP16
    // tensor-core MMAs (mma.sync m16n8k16, FP32 accumulate), 16 positions at a
    // time. K runs over the patch rows padded to 6 (15 pairs, and one of
    // zeros): an A register is two adjacent luma values, one aligned 32-bit
    // load from the copy of the tile that suits the position's parity. The
    // padding is masked, not only multiplied by 0. B fragments (basis, k x n,
    // "col" layout): rows 2t, 2t+1, 2t+8, 2t+9 of column g, per k-step
    uint32_t bf[2][2], mask[4];
    int off[4];
#pragma unroll
    for (int n = 0; n < 4; n++) {
        const int pr = 4 * n + t, dy = pr / 3, j = pr % 3;  // the lane's pairs t, 4 + t, 8 + t, 12 + t
        const bool in = pr < 15;
        off[n] = in ? 2 * (dy * BX_LW + 2 * j) : 0;  // bytes
        mask[n] = in ? (j == 2 ? 0x0000ffffu : 0xffffffffu) : 0u;
        const float b0 = in ? sm.bsm[5 * dy + 2 * j][g] : 0.f, b1 = in && j < 2 ? sm.bsm[5 * dy + 2 * j + 1][g] : 0.f;
        bf[n >> 1][n & 1] = h2u(__floats2half2_rn(b0, b1));
    }
    __syncthreads();
    uint32_t* q32 = reinterpret_cast<uint32_t*>(sm.q);  // [position][4] half2
    const float cen0 = sm.cen[2 * t], cen1 = sm.cen[2 * t + 1];
    float nmax = 0.f;
    // window positions that lie outside the image take its edge's patches
    const bool inner = x0 >= 10 && y0 >= 10 && x0 + BX_W - 10 <= img.w && y0 + T::H - 10 <= img.h;
    int mx[2], my[2];  // window column and row of this thread's two positions of a chunk
#pragma unroll
    for (int e = 0; e < 2; e++) {
        mx[e] = (warp * 16 + g + 8 * e) % BX_W;
        my[e] = (warp * 16 + g + 8 * e) / BX_W;
    }
    const uint32_t luma0 = uint32_t(__cvta_generic_to_shared(sm.luma[0]));
    for (int ch = warp; ch < NPOS / 16; ch += TY) {
        const int m0 = ch * 16 + g, m1 = m0 + 8;  // the two rows of this thread
        // first pair of the patch in the luma tile, around the clamped image
        // position of the window position, as a clamped read of a projected
        // plane would see
        auto first = [&](int e) {
            int px = mx[e], py = my[e];
            if (!inner) {
                px = clampi(x0 - 10 + px, 0, img.w - 1) - (x0 - 10);
                py = clampi(y0 - 10 + py, 0, img.h - 1) - (y0 - 10);
            }
            mx[e] += 16 * TY % BX_W;  // on to the next chunk
            my[e] += 16 * TY / BX_W;
            if (mx[e] >= BX_W) mx[e] -= BX_W, my[e]++;
            // odd columns: the second copy, one half lower
            return luma0 + uint32_t((px & 1) * (T::LH * BX_LW - 1) + py * BX_LW + px) * 2;
        };
        const uint32_t l0 = first(0), l1 = first(1);
        auto av = [&](uint32_t l, int n) {
            uint32_t v;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(l + off[n]));
            return v & mask[n];
        };
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < 2; s++) {
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                "{%0,%1,%2,%3};"
                : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                : "r"(av(l0, 2 * s)), "r"(av(l1, 2 * s)), "r"(av(l0, 2 * s + 1)), "r"(av(l1, 2 * s + 1)),
                  "r"(bf[s][0]), "r"(bf[s][1]));
        }
        // rows m0 (c0, c1) and m1 (c2, c3), components 2t, 2t+1; centre, round, store
        const __half2 h0 = __floats2half2_rn(c[0] - cen0, c[1] - cen1);
        const __half2 h1 = __floats2half2_rn(c[2] - cen0, c[3] - cen1);
        q32[m0 * 4 + t] = h2u(h0);
        q32[m1 * 4 + t] = h2u(h1);
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        float n0 = f0.x * f0.x + f0.y * f0.y, n1 = f1.x * f1.x + f1.y * f1.y;
        n0 += __shfl_xor_sync(0xffffffffu, n0, 1);
        n0 += __shfl_xor_sync(0xffffffffu, n0, 2);
        n1 += __shfl_xor_sync(0xffffffffu, n1, 1);
        n1 += __shfl_xor_sync(0xffffffffu, n1, 2);
        n0 *= 0.5f;
        n1 *= 0.5f;
        if (t == 0) {
            sm.nn[m0] = make_float2(n0, n0);
            sm.nn[m1] = make_float2(n1, n1);
        }
        nmax = fmaxf(nmax, n0 + n1);
        bad = bad || !(n0 + n1 < inf);
    }
    {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(nmax));  // not negative
        if (lane == 0) atomicMax(&sm.nn_max, m);
    }
    __syncthreads();
    // the pixels' constants, once each
    float kmax = 0.f;
    for (int i = tid; i < T::ROWS * BX_TX; i += NT) {
        const int px = i % BX_TX, py = i / BX_TX;
        const int c = (py + 10) * BX_W + px + 10;
        const float4 yb = sm.yb[c];
        const float cr = sm.cr[c].x;
        const BmConst k =
            bm_const<__half>(a, grad, img.w, img.h, min(x0 + px, img.w - 1), min(y0 + py, img.h - 1), yb.x);
        const float kl = 2.f * fmaxf(-2.f * kLog2e * k.s * k.s, -1e30f), sq = sqrtf(lk);
        const float c1 = sq * k.c1, c2 = sq * k.c2;
        sm.k[BK_KL][i] = kl;
        sm.k[BK_BASE][i] = fmaf(kl, sm.nn[c].x, 0.5f * log2f(lk));
        sm.k[BK_C1][i] = c1;
        sm.k[BK_C2][i] = c2;
        sm.k[BK_NO1][i] = -c1 * yb.z;
        sm.k[BK_NO2][i] = -c2 * cr;
        kmax = fmaxf(kmax, -kl);
        bad = bad || !(kl <= 0.f);
    }
    {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(kmax));
        if (lane == 0) atomicMax(&sm.kl_max, m);
    }
    const bool safe = __syncthreads_or(bad);
    // S is not negative but for the rounding of its terms, below 2^-18 of the
    // largest |q'|^2: the exponents stay below log2 sqrt(lk) + 1 < 2 unasked
    // unless the tile's kl are extreme
    const bool clamp = !(__uint_as_float(sm.nn_max) * __uint_as_float(sm.kl_max) < 0x1p18f);
    if (safe) bm_groups<true, true, TY>(sm, part, parts);
    else if (clamp) bm_groups<false, true, TY>(sm, part, parts);
    else bm_groups<false, false, TY>(sm, part, parts);
    __syncthreads();
    for (int i = tid; i < T::ROWS * BX_TX; i += NT) {
        const int x = x0 + i % BX_TX, y = y0 + i / BX_TX;
        if (x >= out.w || y >= out.h) continue;
        // the group's round: another part's pixels still hold their constants
        if ((i / (2 * BX_TX) * (BX_TX / 4) + i % BX_TX / 4) / TY % parts != part) continue;
        const float ny = sm.k[3][i], nc = sm.k[4][i];
        // sums that vanish: at scales where the distance's rounding alone
        // exceeds the exponent's range even the pixel's own weight is lost
        const int c = (i / BX_TX + 10) * BX_W + i % BX_TX + 10;
        const float vy = ny != 0.f ? sm.k[0][i] / ny : sm.yb[c].x;
        const float vb = nc != 0.f ? sm.k[1][i] / nc : sm.yb[c].z, vr = nc != 0.f ? sm.k[2][i] / nc : sm.cr[c].x;
        st4<__half>(out.px(x, y), f4{vy, vb, vr, ny});
    }
}

template <int TY, int NP>
__global__ void __launch_bounds__(BxTile<TY, NP>::THREADS, BxTile<TY, NP>::MIN_BLOCKS)
    k_block_match_pair(Plane<__half, 4> img, Plane<__half, 2> grad, const float* __restrict__ basis,
                       Plane<__half, 4> out, BlockMatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bm_tile<TY, NP>(blockIdx.x * BX_TX, blockIdx.y * (NP * TY), img, grad, basis, out, a,
                    *reinterpret_cast<BmTileSmem<TY, NP>*>(smem_raw), blockIdx.z, gridDim.z);
}

template <int TY, int NP>
static void launch_pair(Plane<__half, 4> img, Plane<__half, 2> grad, const float* basis, Plane<__half, 4> out,
                        const BlockMatchArgs& a, cudaStream_t s, bool split = false) {
    const size_t smem = sizeof(BmTileSmem<TY, NP>);
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_block_match_pair<TY, NP>), int(smem));
    dim3 g((img.w + BX_TX - 1) / BX_TX, (img.h + NP * TY - 1) / (NP * TY));
    // A level too small for the 296 blocks that fit the chip: each tile's groups
    // are dealt to up to 8 blocks, which stage it alike. 126x94 (24 tiles) 20 us,
    // 43 with a block a tile; 256x192 (96) 34 and 44 (41 over two blocks); taken
    // further, past the blocks that fit, 52. A batch's streams share the chip, but
    // seldom more than two are at such a level at once: twelve 256x192 frames on six
    // streams 761 us, 849 if each level counts as alone, 826 with a block a tile,
    // 793 if all six count; two frames 272, 272, 329, 286.
    if (split)
        for (const unsigned z : {2u, 3u, 4u, 8u})  // 4, 3, 2, 1 of a tile's 8 rounds of groups
            if (g.x * g.y * z * unsigned(a.streams) <= 296u * unsigned(a.streams > 2 ? 2 : a.streams)) g.z = z;
    k_block_match_pair<TY, NP><<<g, BxTile<TY, NP>::THREADS, smem, s>>>(img, grad, basis, out, a);
}

// the variants by code (10 TY + NP)
static constexpr int kBmVariants[4] = {84, 44, 82, 162};

static void launch_pair_variant(int code, Plane<__half, 4> img, Plane<__half, 2> grad, const float* basis,
                                Plane<__half, 4> out, const BlockMatchArgs& a, cudaStream_t s) {
    switch (code) {
        case 44: launch_pair<4, 4>(img, grad, basis, out, a, s); break;
        case 82: launch_pair<8, 2>(img, grad, basis, out, a, s, true); break;
        case 162: launch_pair<16, 2>(img, grad, basis, out, a, s); break;
        default: launch_pair<8, 4>(img, grad, basis, out, a, s); break;
    }
}

// ============================================================ FP16-storage path, tensor-core form
// The window sums as matrix products on the tensor cores, one warp per
// group of 16 pixels (a 4 x 4 block, the block shape whose windows overlap
// most: their union is 24 x 24 positions, of which each pixel's 21 x 21
// window is 76.6%). The union is walked as 72 tiles of 8 neighbours (24
// rows x 3 row segments). Per tile:
//   * S = -2 p'.q' + |q'|^2 for the 16 pixels x 8 neighbours by one
//     mma.sync m16n8k8 (FP16 in, FP32 accumulate): A holds each pixel's
//     centred coefficients times -2, B the neighbours' centred
//     coefficients, C the neighbours' |q'|^2. The coefficients are stored
//     in FP16 and the scaling by -2 is exact, so the products are exact
//     and the sum is an FP32 sum, as in a scalar FP32 evaluation;
//   * the weights from the accumulator fragment, two neighbours of a pixel
//     at a time: luma exponent kl S + (kl |p'|^2 + log2 sqrt(lk)) by one
//     packed FP32 FMA, both exponentials as ex2.approx.f16x2 (the
//     reference evaluates its weights in half precision,
//     demosaic.metal:851-874), chroma exponent in packed FP32;
//   * the weights, already in the accumulator layout of S, are the A
//     operand of two more MMAs (two tiles per k-step) against B = the
//     neighbours' (Y, 0, 0, 1) and (0, Cb, Cr, 0, 1) columns, which add
//     sum w Y, sum w Cb, sum w Cr and both kernel norms in FP32.
// A neighbour outside a pixel's window has spatial weight 0 (and
// -log2 weight +inf), which zeroes both of its weights. The spatial
// Gaussian is separable: its x part per lane and row segment is held in
// registers, its y part per union row comes from a 27-entry table.
constexpr int BM_T = 32, BM_W = BM_T + 20, BM_N = BM_W * BM_W, BM_LW = BM_W + 4, BM_THREADS = 256;

struct BmMmaSmem {
    uint4 q[BM_N];               // q - c, 8 halves
    float nn[BM_N];              // |q - c|^2
    __half y[BM_N], cb[BM_N], cr[BM_N];
    float lswy[32];              // -log2 of the spatial weight's y part, dy = -13..13 (+inf outside +-10)
    __half swy[32];              // its y part / sqrt(lk) (0 outside)
    __half luma[BM_LW * BM_LW];  // the luma tile of the projection patches, origin (x0 - 12, y0 - 12)
    float cen[8];                // the centring vector
    float bsm[25][8];            // the level's basis
};

__device__ __forceinline__ uint32_t cvt_h2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t ex2_h2(uint32_t x) {
    uint32_t r;
    asm("ex2.approx.f16x2 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ u64 h2_to_f2(uint32_t h) {
    const float2 f = __half22float2(u2h_(h));
    return pk2(f.x, f.y);
}
__device__ __forceinline__ uint32_t hmin2_u(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void mma16816_acc(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Per pixel row of a lane (pixel g or g + 8 of the group): the constants
// of its two neighbours' weights, as packed pairs.
struct BmRow {
    u64 kl, base;          // luma exponent kl S + base
    u64 c1, c2, no1, no2;  // chroma: d = c v - o
};

// The weights of one pixel row for the lane's two neighbours of a tile:
// (wy, wc) as half2 pairs, from its S pair (s0, s1).
__device__ __forceinline__ void bm_weights(const BmRow& R, float s0, float s1, u64 cbf, u64 crf, u64 lsw,
                                           uint32_t swp, uint32_t& wy, uint32_t& wc) {
    float e0, e1;
    upk2(fma2(R.kl, pk2(s0, s1), R.base), e0, e1);
    // sqrt(lk) lw for both neighbours; the exponent is at most log2 sqrt(lk)
    // but for rounding, and is held below 2 as the FP32 kernel holds it
    const uint32_t lws = ex2_h2(hmin2_u(cvt_h2(e0, e1), 0x40004000u));
    const u64 lf = h2_to_f2(lws);
    const u64 d1 = fma2(R.c1, cbf, R.no1), d2 = fma2(R.c2, crf, R.no2);
    float q0, q1;
    upk2(fma2(lf, lf, fma2(d1, d1, fma2(d2, d2, lsw))), q0, q1);
    wc = ex2_h2(cvt_h2(-q0, -q1));                    // sw cw
    wy = hmul2_u(lws, swp);                           // sw lw
}

// One 32 x 32 tile (origin x0, y0) by a block of BM_THREADS threads.
__device__ __forceinline__ void bm_mma_tile(int x0, int y0, const Plane<__half, 4>& img, const Plane<__half, 2>& grad,
                                            const float* __restrict__ basis, const Plane<__half, 4>& out,
                                            const BlockMatchArgs& a, BmMmaSmem& sm) {
    float* cen = sm.cen;
    float (*bsm)[8] = sm.bsm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const float kLog2e = 1.4426950408889634f, lk = 2.f * kLog2e, isq = rsqrtf(lk);
    // ---- staging: spatial y table, basis, luma tile, Y/Cb/Cr of the window region
    if (tid < 32) {
        const int dy = tid - 13;
        const bool in = dy >= -10 && dy <= 10;
        const float w = in ? spatial_weight(0, dy) : 0.f;
        sm.lswy[tid] = in ? -log2f(w) : __int_as_float(0x7f800000);
        sm.swy[tid] = __float2half_rn(w * isq);
    }
    for (int k = tid; k < 200; k += BM_THREADS) bsm[k / 8][k % 8] = basis[k];
    for (int k = tid; k < BM_LW * BM_LW; k += BM_THREADS) {
        const int ty = k / BM_LW, tx = k % BM_LW;
        sm.luma[k] = *img.pxc(x0 - 12 + tx, y0 - 12 + ty);
    }
    for (int k = tid; k < BM_N; k += BM_THREADS) {
        const int ty = k / BM_W, tx = k % BM_W;
        const __half* p = img.pxc(x0 - 10 + tx, y0 - 10 + ty);
        sm.y[k] = p[0];
        sm.cb[k] = p[1];
        sm.cr[k] = p[2];
    }
    __syncthreads();
    if (tid < 8) {  // centring vector: the coefficients (FP32) of the tile's centre pixel
        const int cx = BM_T / 2 + 12, cy = BM_T / 2 + 12;
        float c = 0.f;
        for (int k = 0; k < 25; k++) c += bsm[k][tid] * __half2float(sm.luma[(cy + k / 5 - 2) * BM_LW + cx + k % 5 - 2]);
        cen[tid] = c;
    }
    // pcaProjection (demosaic.metal:774-796) of every staged position:
    // 16 positions x 5x5 patch (K = 25 padded to 32) x 25x8 basis per MMA
    uint32_t bf[2][2];
#pragma unroll
    for (int s = 0; s < 2; s++) {
        auto bk = [&](int k) { return k < 25 ? bsm[k][g] : 0.f; };
        const int k0 = 16 * s + 2 * t;
        bf[s][0] = h2u(__floats2half2_rn(bk(k0), bk(k0 + 1)));
        bf[s][1] = h2u(__floats2half2_rn(bk(k0 + 8), bk(k0 + 9)));
    }
    __syncthreads();
    uint32_t* q32 = reinterpret_cast<uint32_t*>(sm.q);  // [position][4] half2
    for (int ch = warp; ch < BM_N / 16; ch += BM_THREADS / 32) {
        const int m0 = ch * 16 + g, m1 = m0 + 8;
        auto lidx = [&](int m) {  // the clamped image position of window position m, in the luma tile
            const int px = clampi(x0 - 10 + m % BM_W, 0, img.w - 1) - (x0 - 12);
            const int py = clampi(y0 - 10 + m / BM_W, 0, img.h - 1) - (y0 - 12);
            return py * BM_LW + px;
        };
        const int l0 = lidx(m0), l1 = lidx(m1);
        auto av = [&](int l, int k) { return k < 25 ? sm.luma[l + (k / 5 - 2) * BM_LW + (k % 5 - 2)] : __float2half(0.f); };
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int k0 = 16 * s + 2 * t;
            mma16816_acc(c, h2u(__halves2half2(av(l0, k0), av(l0, k0 + 1))), h2u(__halves2half2(av(l1, k0), av(l1, k0 + 1))),
                         h2u(__halves2half2(av(l0, k0 + 8), av(l0, k0 + 9))),
                         h2u(__halves2half2(av(l1, k0 + 8), av(l1, k0 + 9))), bf[s][0], bf[s][1]);
        }
        const __half2 h0 = __floats2half2_rn(c[0] - cen[2 * t], c[1] - cen[2 * t + 1]);
        const __half2 h1 = __floats2half2_rn(c[2] - cen[2 * t], c[3] - cen[2 * t + 1]);
        q32[m0 * 4 + t] = h2u(h0);
        q32[m1 * 4 + t] = h2u(h1);
        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
        float n0 = f0.x * f0.x + f0.y * f0.y, n1 = f1.x * f1.x + f1.y * f1.y;
        n0 += __shfl_xor_sync(0xffffffffu, n0, 1);
        n0 += __shfl_xor_sync(0xffffffffu, n0, 2);
        n1 += __shfl_xor_sync(0xffffffffu, n1, 1);
        n1 += __shfl_xor_sync(0xffffffffu, n1, 2);
        if (t == 0) {
            sm.nn[m0] = n0;
            sm.nn[m1] = n1;
        }
    }
    __syncthreads();

    // ---- lane constants: the x part of the spatial weight for the lane's
    //      neighbour pair (2t, 2t + 1) of each row segment, pixel column g % 4
    const int pxl = g & 3;
    u64 lswx[3];
    uint32_t swx[3];
#pragma unroll
    for (int s = 0; s < 3; s++) {
        float l[2], w[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int dx = 8 * s + 2 * t + e - pxl - 10;
            const bool in = dx >= -10 && dx <= 10;
            w[e] = in ? spatial_weight(dx, 0) : 0.f;
            l[e] = in ? -log2f(w[e]) : __int_as_float(0x7f800000);
        }
        lswx[s] = pk2(l[0], l[1]);
        swx[s] = cvt_h2(w[0], w[1]);
    }
    const uint32_t ONE2 = 0x3c003c00u;  // half2 (1, 1)
    const __half* ysrc = sm.y;  // the luma B column (lanes g == 0)

    // ---- 4 x 4 pixel groups: 64 per tile, warp w takes groups w, w + 8, ...
    for (int grp = warp; grp < (BM_T / 4) * (BM_T / 4); grp += BM_THREADS / 32) {
        const int gx = (grp % (BM_T / 4)) * 4, gy = (grp / (BM_T / 4)) * 4;  // tile coordinates
        // the lane's two pixels: rows g and g + 8 of the group = (g % 4, g / 4) and (g % 4, g / 4 + 2)
        BmRow R[2];
        uint32_t ap[2];  // A fragments: -2 p', components 2t, 2t + 1
        int py[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            py[r] = (g >> 2) + 2 * r;
            const int sx = gx + pxl + 10, sy = gy + py[r] + 10;  // staged position of the pixel
            const int pos = sy * BM_W + sx;
            const float in_y = __half2float(sm.y[pos]), in_cb = __half2float(sm.cb[pos]), in_cr = __half2float(sm.cr[pos]);
            const int ix = min(x0 + gx + pxl, img.w - 1), iy = min(y0 + gy + py[r], img.h - 1);
            const BmConst k = bm_const<__half>(a, grad, img.w, img.h, ix, iy, in_y);
            const float kl = fmaxf(-2.f * kLog2e * k.s * k.s, -1e30f);
            const float base = fmaf(kl, sm.nn[pos], 0.5f * log2f(lk));
            const float sq = sqrtf(lk);
            const float c1 = sq * k.c1, c2 = sq * k.c2;
            R[r].kl = pk2(kl, kl);
            R[r].base = pk2(base, base);
            R[r].c1 = pk2(c1, c1);
            R[r].c2 = pk2(c2, c2);
            R[r].no1 = pk2(-c1 * in_cb, -c1 * in_cb);
            R[r].no2 = pk2(-c2 * in_cr, -c2 * in_cr);
            ap[r] = hmul2_u(q32[pos * 4 + t], 0xc000c000u);  // p' components 2t, 2t + 1, times -2 (exact)
        }
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        // union rows ny = 0..23 (staged rows gy + ny), segments s = 0..2
        // (staged columns gx + 8 s .. + 7): tiles in row-major order, two per k-step
        uint32_t pwy[2], pwc[2], pby, pbc;  // the pending (first) tile of a k-step
#pragma unroll 1
        for (int ny = 0; ny < 24; ny += 2) {
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const int row = ny + j / 3, s = j % 3;
                const int base_pos = (gy + row) * BM_W + gx + 8 * s;
                // B of S: neighbour g's coefficients 2t, 2t + 1
                const uint32_t bq = q32[(base_pos + g) * 4 + t];
                const float2 nnp = *reinterpret_cast<const float2*>(&sm.nn[base_pos + 2 * t]);
                float S[4];
                mma1688(S, ap[0], ap[1], bq, nnp.x, nnp.y, nnp.x, nnp.y);
                const uint32_t cbh = *reinterpret_cast<const uint32_t*>(&sm.cb[base_pos + 2 * t]);
                const uint32_t crh = *reinterpret_cast<const uint32_t*>(&sm.cr[base_pos + 2 * t]);
                const uint32_t yh = *reinterpret_cast<const uint32_t*>(&ysrc[base_pos + 2 * t]);
                const u64 cbf = h2_to_f2(cbh), crf = h2_to_f2(crh);
                uint32_t wy[2], wc[2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int dyi = row - py[r] - 10 + 13;  // 0..26
                    const float ly = sm.lswy[dyi];
                    const __half sy = sm.swy[dyi];
                    const u64 lsw = add2(lswx[s], pk2(ly, ly));
                    const uint32_t swp = hmul2_u(swx[s], h2u(__halves2half2(sy, sy)));
                    bm_weights(R[r], S[2 * r], S[2 * r + 1], cbf, crf, lsw, swp, wy[r], wc[r]);
                }
                // B columns of the sums: luma (Y, 0, 0, 1, 0..), chroma (0, Cb, Cr, 0, 1, 0..)
                const uint32_t by = g == 0 ? yh : (g == 3 ? ONE2 : 0u);
                const uint32_t bc = g == 1 ? cbh : (g == 2 ? crh : (g == 4 ? ONE2 : 0u));
                if ((j & 1) == 0) {
                    pwy[0] = wy[0]; pwy[1] = wy[1]; pwc[0] = wc[0]; pwc[1] = wc[1]; pby = by; pbc = bc;
                } else {
                    mma16816_acc(acc, pwy[0], pwy[1], wy[0], wy[1], pby, by);
                    mma16816_acc(acc, pwc[0], pwc[1], wc[0], wc[1], pbc, bc);
                }
            }
        }
        // acc: rows g, g + 8; columns 2t, 2t + 1. Column 0 sum wy Y, 1 sum wc Cb,
        // 2 sum wc Cr, 3 sum wy, 4 sum wc: gather to lane t = 0
        const float a2 = __shfl_down_sync(0xffffffffu, acc[0], 1), a3 = __shfl_down_sync(0xffffffffu, acc[1], 1);
        const float a4 = __shfl_down_sync(0xffffffffu, acc[0], 2);
        const float b2 = __shfl_down_sync(0xffffffffu, acc[2], 1), b3 = __shfl_down_sync(0xffffffffu, acc[3], 1);
        const float b4 = __shfl_down_sync(0xffffffffu, acc[2], 2);
        if (t == 0) {
            const int ox = x0 + gx + pxl;
            if (ox < out.w) {
                const int oy0 = y0 + gy + py[0], oy1 = y0 + gy + py[1];
                if (oy0 < out.h) st4<__half>(out.px(ox, oy0), f4{acc[0] / a3, acc[1] / a4, a2 / a4, a3});
                if (oy1 < out.h) st4<__half>(out.px(ox, oy1), f4{acc[2] / b3, acc[3] / b4, b2 / b4, b3});
            }
        }
    }
}

__global__ void __launch_bounds__(BM_THREADS, 2)
    k_block_match_mma(Plane<__half, 4> img, Plane<__half, 2> grad, const float* __restrict__ basis,
                      Plane<__half, 4> out, BlockMatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bm_mma_tile(blockIdx.x * BM_T, blockIdx.y * BM_T, img, grad, basis, out, a,
                *reinterpret_cast<BmMmaSmem*>(smem_raw));
}

static void launch_mma(Plane<__half, 4> img, Plane<__half, 2> grad, const float* basis, Plane<__half, 4> out,
                       const BlockMatchArgs& a, cudaStream_t s) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_block_match_mma), int(sizeof(BmMmaSmem)));
    dim3 g((img.w + BM_T - 1) / BM_T, (img.h + BM_T - 1) / BM_T);
    k_block_match_mma<<<g, BM_THREADS, sizeof(BmMmaSmem), s>>>(img, grad, basis, out, a);
}

// ============================================================ persistent batch kernel
// PyramidProcessor::denoise (pyramid_processor.cpp:96-172) for every frame
// of a batch in one launch. The host lists the work of every (frame,
// level) as tasks: reconstruct tiles (SN, 64 x 64 pixels), covariance
// partial rows (COV), the eigen-solve (EIG) and block-matching tiles (BM,
// 32 x 32), level by level from the coarsest, all frames' SN / COV / EIG of
// a level before their BM tiles. A block takes the next task from a
// counter, waits until the task's inputs are complete, runs it with the
// same device code as the stream kernels (so the results are
// bit-identical), and counts it done:
//   SN (f, l)  waits for every BM tile of (f, l + 1)  (the coarse denoised image)
//   COV (f, l) waits for every SN tile of (f, l)      (the layer)
//   EIG (f, l) waits for every COV row of (f, l)     (without patches, for its SN tiles)
//   BM (f, l)  waits for EIG (f, l)                   (the basis; the layer before it)
// Every task a block waits for comes earlier in the list and was taken by a
// running block, so the earliest unfinished task can always run: the order
// cannot deadlock, and the blocks need not be co-resident. A wait is
// bounded: past limit_ns (global timer) the block records the task type
// in *err and every block stops taking tasks; the host reads the word and
// returns GLS_ERR_TIMEOUT.
struct PSmem {
    union {
        BmTileSmem<8, 2> bm;  // a 32 x 16 tile
        EigenSmem eig;
        CovSmem cov;
    };
};

__device__ __forceinline__ long long global_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The two calls below take the block's shared memory from the extern
// array itself, not as a pointer argument: across a call boundary a pointer
// is generic, and the tile's staged reads would compile to generic loads
// instead of shared-memory loads. Their level arguments are copied out of
// the descriptor once, as a kernel's parameters would be.

// the rarely taken eigen-solve as a call of its own, so that its registers
// do not weigh on the block-matching path
__device__ __noinline__ void persistent_eigen(const PLevel& L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pca_eigen_block(L.part, L.n_cov, (L.layer.w / 8) * (L.layer.h / 8), L.basis, L.status,
                    reinterpret_cast<PSmem*>(smem_raw)->eig);
}

// a block-matching task: one 32 x 16 tile of the default matcher by the
// block's 8 warps, the same bits as every stream variant
__device__ __noinline__ void persistent_bm(const PLevel& L, uint32_t item) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Plane<__half, 4> layer = L.layer, den = L.den;
    const Plane<__half, 2> grad = L.grad;
    const float* basis = L.basis;
    const BlockMatchArgs ba = L.ba;
    const int tx = int(item) % L.tiles_x, ty = int(item) / L.tiles_x;
    bm_tile<8, 2>(tx * BX_TX, ty * kPBmRows, layer, grad, basis, den, ba, reinterpret_cast<PSmem*>(smem_raw)->bm);
}

__global__ void __launch_bounds__(BM_THREADS, 2)
    k_pyramid_persistent(const PTask* __restrict__ tasks, int n_tasks, const PLevel* __restrict__ lv,
                         PCounters* __restrict__ cnt, int* __restrict__ next, int* __restrict__ err, long long limit_ns) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PSmem& sm = *reinterpret_cast<PSmem*>(smem_raw);
    __shared__ int s_task, s_ok;
    for (;;) {
        if (threadIdx.x == 0) s_task = ld_acquire(err) ? n_tasks : atomicAdd(next, 1);
        __syncthreads();
        const int ti = s_task;
        if (ti >= n_tasks) break;
        const PTask tk = tasks[ti];
        const uint32_t type = tk.item >> 30, item = tk.item & kPTaskItemMask;
        const PLevel& L = lv[tk.lev];
        if (threadIdx.x == 0) {
            // the counter this task waits on and its target (none: -1)
            const int* c = nullptr;
            int target = 0;
            if (type == PT_SN) {
                c = &cnt[L.coarser].bm;
                target = lv[L.coarser].n_bm;
            } else if (type == PT_COV) {
                if (L.n_sn > 0) {
                    c = &cnt[tk.lev].sn;
                    target = L.n_sn;
                }
            } else if (type == PT_EIG) {  // a level without patches has no row: its layer has to be there for BM
                c = L.n_cov > 0 || L.n_sn == 0 ? &cnt[tk.lev].cov : &cnt[tk.lev].sn;
                target = L.n_cov > 0 || L.n_sn == 0 ? L.n_cov : L.n_sn;
            } else {
                c = &cnt[tk.lev].eig;
                target = 1;
            }
            int ok = 1;
            if (c && ld_acquire(c) < target) {
                const long long t0 = global_ns();
                unsigned ns = 32;
                while (ld_acquire(c) < target) {
                    if (ld_acquire(err) || global_ns() - t0 > limit_ns) {
                        atomicCAS(err, 0, int(1 + type));
                        ok = 0;
                        break;
                    }
                    __nanosleep(ns);
                    ns = ns < 2048 ? 2 * ns : ns;
                }
            }
            __threadfence();
            s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) break;
        int* done;
        if (type == PT_SN) {
            const int tx = item % L.sn_tiles_x, ty = item / L.sn_tiles_x;
            for (int k = threadIdx.x; k < kPSnTile * kPSnTile; k += BM_THREADS) {
                const int x = tx * kPSnTile + k % kPSnTile, y = ty * kPSnTile + k / kPSnTile;
                if (x < L.img.w && y < L.img.h)
                    subtract_noise_px<__half>(L.img, L.coarse, L.coarse_den, L.grad, L.layer, L.sa, L.rx, L.ry, x, y);
            }
            done = &cnt[tk.lev].sn;
        } else if (type == PT_COV) {
            const int c0 = int(item) * L.cov_group;
            pca_cov_row<__half>(L.layer, L.part + size_t(item) * kPcaAcc, c0, min(c0 + L.cov_group, L.chunks), sm.cov);
            done = &cnt[tk.lev].cov;
        } else if (type == PT_EIG) {
            persistent_eigen(L);
            done = &cnt[tk.lev].eig;
        } else {
            persistent_bm(L, item);
            done = &cnt[tk.lev].bm;
        }
        __syncthreads();  // the task's writes, and its shared memory, are finished
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(done, 1);
        }
    }
}

int persistent_grid(int device) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_pyramid_persistent), int(sizeof(PSmem)));
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pyramid_persistent, BM_THREADS, sizeof(PSmem)) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return 0;
    return per_sm * sms;
}

void launch_pyramid_persistent(const PTask* tasks, int n, const PLevel* lv, PCounters* cnt, int* next, int* err,
                               long long limit_ns, int grid, cudaStream_t s) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_pyramid_persistent), int(sizeof(PSmem)));
    k_pyramid_persistent<<<grid, BM_THREADS, sizeof(PSmem), s>>>(tasks, n, lv, cnt, next, err, limit_ns);
}

// The tile variant of the FP16 block matcher. The variants (warps x pixels per
// lane: 8 x 4 and 16 x 2 for 32 x 32 tiles, 4 x 4 and 8 x 2 for 32 x 16)
// compute identical results (a pixel's group, its walk and its centring are
// the same), so the choice only changes speed. 8 x 2 is taken for every size:
// two of its blocks share an SM, so one stages while the other computes. A
// 32 x 32 tile stages 28% fewer positions per pixel but fills an SM alone:
// 16 x 2 takes 2.26 ms a 2016x1512 denoise against 2.09, 48.5 ms a batch of six
// 12 MP frames against 46.2, 0.385 ms a 256x192 frame against 0.314; 8 x 4 and
// 4 x 4 hold half the warps (2.61 and 2.55 ms). GLS_BM_TILE=84, 44, 82 or 162
// in the environment (or 8 / 4 for 84 / 44) fixes the variant. The level sizes
// met are listed for gls_block_match_tiles; host threads that drive converters
// of their own share the lock.
static std::shared_mutex g_tile_mu;
static std::map<std::pair<int, int>, int> g_tile_choice;

int bm_tile_list(int* whty, int max) {
    std::shared_lock<std::shared_mutex> lk(g_tile_mu);
    int n = 0;
    for (const auto& kv : g_tile_choice) {
        if (n < max) {
            whty[3 * n] = kv.first.first;
            whty[3 * n + 1] = kv.first.second;
            whty[3 * n + 2] = kv.second;
        }
        n++;
    }
    return n;
}

static int bm_tile_variant(int w, int h) {
    static const int variant = [] {
        const char* e = std::getenv("GLS_BM_TILE");
        const int v = e ? std::atoi(e) : 0;
        if (v == 8) return 84;  // the thread-row counts of the two NP = 4 variants
        if (v == 4) return 44;
        for (int c : kBmVariants)
            if (v == c) return v;
        return 82;
    }();
    {
        std::shared_lock<std::shared_mutex> lk(g_tile_mu);
        if (g_tile_choice.count({w, h})) return variant;
    }
    std::unique_lock<std::shared_mutex> lk(g_tile_mu);
    g_tile_choice.emplace(std::make_pair(w, h), variant);
    return variant;
}

template <int NP>
static void launch_plain(Plane<float, 4> img, Plane<float, 2> grad, Plane<float, 8> pca, Plane<float, 4> out,
                         const BlockMatchArgs& a, cudaStream_t s) {
    using T = BmPlainTile<NP>;
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_block_match_plain<NP>), int(sizeof(typename T::Smem)));
    const dim3 g((img.w + T::TX - 1) / T::TX, (img.h + T::ROWS - 1) / T::ROWS);
    k_block_match_plain<NP><<<g, dim3(T::TX, T::TY), sizeof(typename T::Smem), s>>>(img, grad, pca, out, a);
}

template <class S>
void launch_block_match(Plane<S, 4> img, Plane<S, 2> grad, Plane<S, 8> pca, const float* basis, Plane<S, 4> out,
                        const BlockMatchArgs& a, cudaStream_t s) {
    if constexpr (is_half<S>::value) {
        // the default matcher unless the call asks for the one with half-precision
        // weights (GLS_BM_TENSOR) or GLS_BM_KERNEL=mma selects that for the process
        static const bool mma_env = [] {
            const char* e = std::getenv("GLS_BM_KERNEL");
            return e && std::strcmp(e, "mma") == 0;
        }();
        if (a.tensor || mma_env) {
            launch_mma(img, grad, basis, out, a, s);
            return;
        }
        launch_pair_variant(bm_tile_variant(img.w, img.h), img, grad, basis, out, a, s);
    } else {
        // One pixel a thread while its 32 x 4 tiles fit the chip's 148 SMs one
        // each: 128x96 (96 of them) 23 us, 32 with two pixels a thread; at
        // 256x192 (384) both take 47-49 us, at 1024x768 580 and 428.
        if (((img.w + 31) / 32) * ((img.h + 3) / 4) <= 148)
            launch_plain<1>(img, grad, pca, out, a, s);
        else
            launch_plain<2>(img, grad, pca, out, a, s);
    }
}

template void launch_block_match<float>(Plane<float, 4>, Plane<float, 2>, Plane<float, 8>, const float*,
                                        Plane<float, 4>, const BlockMatchArgs&, cudaStream_t);
template void launch_block_match<__half>(Plane<__half, 4>, Plane<__half, 2>, Plane<__half, 8>, const float*,
                                         Plane<__half, 4>, const BlockMatchArgs&, cudaStream_t);

}  // namespace gls
