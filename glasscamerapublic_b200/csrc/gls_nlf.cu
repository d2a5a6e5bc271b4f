// gls_nlf.cu — noise-model measurement of RawConverter with
// calibrateFromImage:
//   * k_raw_stats    basicRawNoiseStatistics (demosaic.metal:1110-1136): the
//                    9x9 mean and variance of the four raw channels at every
//                    half-resolution position, from a shared-memory tile,
//                    and each position's variance class counted into the
//                    fit's histogram
//   * k_ycc_stats    basicNoiseStatistics (:1138-1159): the 5x5 mean of Y
//                    and variances of Y, Cb, Cr at every position of a
//                    level, and their variance classes
//   * k_fit_pass /   the two-pass least-squares fits of MeasureRawNLF
//     k_fit_finish   (raw_converter.cpp:339-490) and MeasureYCbCrNLF
//                    (pyramid_processor.cpp:173-324) on the device: each
//                    pass sums over the statistics in FP64 (fixed grid,
//                    block partial sums in a fixed order, so the result does
//                    not depend on scheduling) and a one-block kernel forms
//                    the fit from the partial sums
// The statistics are FP32 operation for operation as in the reference
// kernels (one rounding per operation, no contraction, each channel's taps
// in the reference's order), so the FP32 path's statistics equal the CPU
// oracle's bit for bit; the fits agree with the oracle's sequential FP64
// sums to their last bits.
#include <type_traits>

#include <cmath>

#include "../../include/glscam.h"
#include "gls_common.cuh"
#include "gls_kernels.h"

namespace gls {

namespace {

// ---------------------------------------------------------------- statistics
// The variance class of a position: 6 + trunc(clamp(log10(v), -6, -1)) of
// its largest variance v (raw_converter.cpp:357-362), taken from the first
// channel on so that a NaN in a later channel never wins. The truncation
// makes the classes (0, 1e-6], (1e-6, 1e-5], (1e-5, 1e-4], (1e-4, 1e-3],
// (1e-3, 1e-2] and above: an FP32 variance lies more than 1e-11 (relative)
// from every power of ten, so the thresholds, rounded down to floats, give
// the logarithm's classes exactly. -1: no class (a NaN; for the YCbCr fit
// also a non-positive variance; a NaN largest value, which the reference
// turns into an undefined histogram index).
template <int N>
__device__ __forceinline__ int variance_class(const float (&v)[N], bool raw) {
    bool valid = true;
#pragma unroll
    for (int c = 0; c < N; c++) valid = valid && !isnan(v[c]) && (raw || v[c] > 0.f);
    if (!valid || v[0] < 0.f) return -1;  // log10 of a negative first variance is NaN
    float m = v[0];                        // 0: log10 = -inf, which any positive variance beats
#pragma unroll
    for (int c = 1; c < N; c++)
        if (v[c] > m) m = v[c];
    // the largest floats below the powers of ten
    constexpr float t6 = 0x1.0c6f7a0000000p-20f, t5 = 0x1.4f8b580000000p-17f, t4 = 0x1.a36e2e0000000p-14f;
    constexpr float t3 = 0x1.0624dc0000000p-10f, t2 = 0x1.47ae140000000p-7f;
    return m <= t6 ? 0 : m <= t5 ? 1 : m <= t4 ? 2 : m <= t3 ? 3 : m <= t2 ? 4 : 5;
}

// a value and its square, added to a sum and a sum of squares at once (packed
// FP32: each lane rounds as the scalar operation)
typedef unsigned long long u64;
__device__ __forceinline__ float2 with_square(float t) { return make_float2(t, __fmul_rn(t, t)); }
__device__ __forceinline__ void add_to(u64& s, u64 t) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s) : "l"(t)); }
__device__ __forceinline__ float2 sums_of(u64 s) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(s));
    return v;
}

constexpr int RS_TX = 32, RS_TY = 8;                         // half-resolution positions per block
constexpr int RS_W = 2 * RS_TX + 10, RS_H = 2 * RS_TY + 10;  // full-resolution tile: 2x + [-4, 5]

// the block's class counts: 8 bits a class in two words, summed over the warp
// (at most 4 positions a lane), one shared atomic per warp and class
struct ClassCount {
    unsigned lo = 0, hi = 0;
    __device__ __forceinline__ void add(int k) {
        if (k >= 0) (k < 4 ? lo : hi) += 1u << (8 * (k & 3));
    }
    __device__ __forceinline__ void flush(unsigned* cls) const {
        const unsigned lane = threadIdx.x & 31;
        // 32 lanes' counts of 4: up to 128
        const unsigned a = __reduce_add_sync(0xffffffffu, lo), b = __reduce_add_sync(0xffffffffu, hi);
        const unsigned n = (lane < 4 ? a : b) >> (8 * (lane & 3)) & 255u;
        if (lane < 6 && n) atomicAdd(&cls[lane], n);
    }
};

// x / D, correctly rounded, in two operations with the reciprocal as a sum of
// two floats (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", 2004; all 2^23
// significands checked for 25 and 81); outside the exponents where the products
// neither overflow nor lose bits, the division itself.
template <int D>
__device__ __forceinline__ float div_const(float x) {
    constexpr float zh = 1.f / float(D), zl = float(1.0 / double(D) - double(zh));
    const float a = fabsf(x);
    if ((a >= 0x1p-90f && a <= 0x1p100f) || a == 0.f) return __fmaf_rn(x, zh, __fmul_rn(x, zl));
    return __fdiv_rn(x, float(D));
}

// PATTERN: the Bayer pattern, so every channel's tap set is known at
// compile time. Bound by the FMA pipe: 648 additions a position whose order is
// fixed, in 324 packed instructions; values are staged with their squares.
// 2016x1512 positions: 109 us (132 with scalar additions, 118 with two
// vertically adjacent positions a thread, which also leaves small frames'
// blocks too few: 128x96 positions 7.1 us, 10.1 with two).
template <class S, int PATTERN>
__global__ void __launch_bounds__(RS_TX* RS_TY) k_raw_stats(Plane<S, 1> raw, Plane<float, 4> mean,
                                                            Plane<float, 4> var, unsigned* __restrict__ hist) {
    constexpr int OX[4][4] = {{1, 0, 0, 1}, {0, 0, 1, 1}, {0, 0, 1, 1}, {1, 0, 0, 1}};
    constexpr int OY[4][4] = {{0, 0, 1, 1}, {1, 0, 0, 1}, {0, 1, 1, 0}, {1, 1, 0, 0}};
    __shared__ __align__(16) float2 tile[RS_H][RS_W];
    __shared__ unsigned cls[6];
    const int X0 = blockIdx.x * RS_TX, Y0 = blockIdx.y * RS_TY;  // half-resolution origin
    const int tid = threadIdx.y * RS_TX + threadIdx.x;
    if (tid < 6) cls[tid] = 0;
    for (int ty = threadIdx.y; ty < RS_H; ty += RS_TY)
        for (int tx = threadIdx.x; tx < RS_W; tx += RS_TX)
            tile[ty][tx] = with_square(to_f(*raw.pxc(2 * X0 - 4 + tx, 2 * Y0 - 4 + ty)));
    __syncthreads();
    const int x = X0 + threadIdx.x, y = Y0 + threadIdx.y;
    // the window steps one full-resolution pixel from 2 (x, y) - 4 and
    // reads each channel at its Bayer offset (readRAWQuad): channel c
    // reads the 10 x 10 block's 9 x 9 sub-block at its offset. Each
    // value is loaded once and added to the channels that read it, each
    // channel still in row-major order of its own taps.
    u64 acc[4] = {};
    const int bx0 = 2 * threadIdx.x, by0 = 2 * threadIdx.y;
#pragma unroll
    for (int r = 0; r < 10; r++)
#pragma unroll
        for (int v = 0; v < 10; v += 2) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&tile[by0 + r][bx0 + v]);
#pragma unroll
            for (int e = 0; e < 2; e++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int j = r - OY[PATTERN][c], i = v + e - OX[PATTERN][c];
                    if (j >= 0 && j < 9 && i >= 0 && i < 9) add_to(acc[c], e ? q.y : q.x);
                }
        }
    ClassCount count;
    if (x < mean.w && y < mean.h) {
        f4 m, vv;
        float* mp = &m.x;
        float* vp = &vv.x;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float2 t = sums_of(acc[c]);
            mp[c] = div_const<81>(t.x);
            vp[c] = div_const<81>(__fsub_rn(t.y, div_const<81>(__fmul_rn(t.x, t.x))));
        }
        st4<float>(mean.px(x, y), m);
        st4<float>(var.px(x, y), vv);
        const float vc[4] = {vv.x, vv.y, vv.z, vv.w};
        count.add(variance_class<4>(vc, true));
    }
    count.flush(cls);
    __syncthreads();
    if (tid < 6 && cls[tid]) atomicAdd(&hist[tid], cls[tid]);
}

// YS_P vertically adjacent positions a thread: a row's values, staged with their
// squares, are read once for the up to YS_P windows that take them. Bound by the FMA pipe
// (150 additions a position whose order is fixed) and 390 MB of traffic.
// 4032x3024: 143 us (224 with one position a thread and scalar squares).
constexpr int YS_TX = 32, YS_TY = 8, YS_W = YS_TX + 4;

template <class S, int YS_P>
__global__ void __launch_bounds__(YS_TX* YS_TY) k_ycc_stats(Plane<S, 4> img, Plane<float, 4> stats,
                                                            unsigned* __restrict__ hist) {
    constexpr int YS_ROWS = YS_TY * YS_P, YS_H = YS_ROWS + 4;
    __shared__ float2 tile[3][YS_H][YS_W];
    __shared__ unsigned cls[6];
    const int x0 = blockIdx.x * YS_TX, y0 = blockIdx.y * YS_ROWS;
    const int tid = threadIdx.y * YS_TX + threadIdx.x;
    if (tid < 6) cls[tid] = 0;
    for (int k = tid; k < YS_W * YS_H; k += YS_TX * YS_TY) {
        const int ty = k / YS_W, tx = k % YS_W;
        const f4 p = ld4<S>(img.pxc(x0 - 2 + tx, y0 - 2 + ty));
        tile[0][ty][tx] = with_square(p.x);
        tile[1][ty][tx] = with_square(p.y);
        tile[2][ty][tx] = with_square(p.z);
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, ty = threadIdx.y * YS_P;
    u64 acc[YS_P][3] = {};
#pragma unroll
    for (int r = 0; r < YS_P + 4; r++)
#pragma unroll
        for (int dx = 0; dx < 5; dx++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const u64 t = *reinterpret_cast<const u64*>(&tile[c][ty + r][threadIdx.x + dx]);
#pragma unroll
                for (int p = 0; p < YS_P; p++)
                    if (r - p >= 0 && r - p < 5) add_to(acc[p][c], t);
            }
    ClassCount count;
#pragma unroll
    for (int p = 0; p < YS_P; p++) {
        const int y = y0 + ty + p;
        if (x >= img.w || y >= img.h) continue;
        f4 o;
        float* op = &o.y;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float2 t = sums_of(acc[p][c]);
            if (c == 0) o.x = div_const<25>(t.x);
            op[c] = div_const<25>(__fsub_rn(t.y, div_const<25>(__fmul_rn(t.x, t.x))));
        }
        st4<float>(stats.px(x, y), o);
        const float vc[3] = {o.y, o.z, o.w};
        count.add(variance_class<3>(vc, false));
    }
    count.flush(cls);
    __syncthreads();
    if (tid < 6 && cls[tid]) atomicAdd(&hist[tid], cls[tid]);
}

// ---------------------------------------------------------------- fits
// raw: mean and var planes, a regressor per channel (4 channels);
// ycc: one statistics plane (mean Y, var Y, Cb, Cr), the luma mean the
// regressor of all three variances
struct FitInput {
    const float4* mean;  // raw: means; ycc: the statistics
    const float4* var;   // raw: variances; ycc: unused
    int w, h;
    size_t pitch;  // float4 per row
    int raw;       // 1: MeasureRawNLF, 0: MeasureYCbCrNLF
    double pixels;  // raw: the raw frame's pixel count; ycc: the level's
    float exposure;
};

constexpr int FIT_BLOCKS = 296, FIT_THREADS = 256, FIT_K = 24;

// one position's regressors and variances (ycc: one regressor, three variances)
template <bool RAW>
struct Sample {
    static constexpr int NM = RAW ? 4 : 1, NV = RAW ? 4 : 3;
    float m[NM], v[NV];
};

template <bool RAW>
__device__ __forceinline__ Sample<RAW> load_sample(const FitInput& in, int x, int y) {
    const size_t i = size_t(y) * in.pitch + x;
    if constexpr (RAW) {
        const float4 m = __ldg(in.mean + i), v = __ldg(in.var + i);
        return {{m.x, m.y, m.z, m.w}, {v.x, v.y, v.z, v.w}};
    } else {
        const float4 t = __ldg(in.mean + i);
        return {{t.x}, {t.y, t.z, t.w}};
    }
}

__device__ __forceinline__ int nch(const FitInput& in) { return in.raw ? 4 : 3; }

// a position counts in the fits: no NaN, every mean in [0.001, 0.9] and
// every variance within the bound (rounded down: the same on FP32 variances;
// likewise 0.001f is the least float above 0.001 and 0.9f the largest below 0.9)
template <bool RAW>
__device__ __forceinline__ bool usable(const Sample<RAW>& s, const float (&bound)[4]) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < s.NM; c++) ok = ok && s.m[c] >= 0.001f && s.m[c] <= 0.9f;
#pragma unroll
    for (int c = 0; c < s.NV; c++) ok = ok && s.v[c] <= bound[c];
    return ok;
}

struct FitState {
    double bound[4];
    double A[4], B[4];
    double err2[4];
    double N1;
};

__device__ __forceinline__ double max_s(double v, double s) { return v > s ? v : s; }

// pass: 1 the first fit's sums; 2 its squared residuals; 3 the second fit's
// sums and squared residuals (the class histogram, pass 0, comes with the
// statistics). Bound by reading the statistics, 97 MB (raw) or 195 MB (YCbCr)
// at 4032x3024 with few warps in flight: four or eight positions a thread are
// loaded before they are summed. Passes 1, 2, 3 of both fits at that size: 64,
// 63, 73 us (180, 164, 149 with one position at a time, a 64-bit division for each and
// the tests in FP64).
template <int PASS, bool RAW>
__global__ void __launch_bounds__(FIT_THREADS, 2) k_fit_pass(FitInput in, const FitState* __restrict__ st_,
                                                          double* __restrict__ partial) {
    constexpr int NK = PASS == 1 ? 17 : PASS == 2 ? 4 : 21, AHEAD = RAW ? 4 : 8;
    using Smp = Sample<RAW>;
    __shared__ double red[FIT_THREADS / 32][NK];
    double acc[NK];
#pragma unroll
    for (int k = 0; k < NK; k++) acc[k] = 0.0;
    const FitState st = *st_;
    float bound[4];
#pragma unroll
    for (int c = 0; c < 4; c++) bound[c] = __double2float_rd(st.bound[c]);
    unsigned count = 0;
    auto add = [&](const Smp& s) {
        if (!usable<RAW>(s, bound)) return;
        if (PASS > 1) {
            double d2[4] = {0.0, 0.0, 0.0, 0.0};
            bool fits = true;
#pragma unroll
            for (int c = 0; c < Smp::NV; c++) {
                const double d = (st.A[c] + st.B[c] * double(s.m[RAW ? c : 0])) - double(s.v[c]);
                d2[c] = d * d;
                fits = fits && (PASS == 2 || d2[c] <= (RAW ? 0.5 : 1.0) * st.err2[c]);
            }
            if (!fits) return;
#pragma unroll
            for (int c = 0; c < Smp::NV; c++) acc[(PASS == 2 ? 0 : 17) + c] += d2[c];
        }
        if (PASS != 2) {
#pragma unroll
            for (int c = 0; c < Smp::NM; c++) {
                const double m = s.m[c];
                acc[c] += m;
                acc[8 + c] += m * m;
            }
#pragma unroll
            for (int c = 0; c < Smp::NV; c++) {
                const double v = s.v[c];
                acc[4 + c] += v;
                acc[12 + c] += double(s.m[RAW ? c : 0]) * v;
            }
            count++;
        }
    };
    constexpr unsigned stride = FIT_BLOCKS * FIT_THREADS;
    const unsigned first = blockIdx.x * FIT_THREADS + threadIdx.x;
    const int step_x = int(stride % unsigned(in.w)), step_y = int(stride / unsigned(in.w));
    int x = int(first % unsigned(in.w)), y = int(first / unsigned(in.w));
    while (y < in.h) {
        Smp s[AHEAD];
        int n = 0;
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            if (y >= in.h) break;
            s[k] = load_sample<RAW>(in, x, y);
            n = k + 1;
            x += step_x;
            y += step_y;
            if (x >= in.w) {
                x -= in.w;
                y++;
            }
        }
#pragma unroll
        for (int k = 0; k < AHEAD; k++)
            if (k < n) add(s[k]);
    }
    if constexpr (PASS != 2) {
        acc[16] = double(count);
        if constexpr (!RAW) {  // the three channels' regressor is one
            acc[1] = acc[2] = acc[0];
            acc[9] = acc[10] = acc[8];
        }
    }
    // block sums in a fixed order: a shuffle tree per warp, then the warps
    // in order
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NK; k++) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < NK) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < FIT_THREADS / 32; w++) t += red[w][threadIdx.x];
        partial[size_t(blockIdx.x) * FIT_K + threadIdx.x] = t;
    }
}

// sums the block partials (a warp per sum: lane-strided blocks, then a
// shuffle tree) and forms the pass's result; pass 0 forms the variance
// bound from the class histogram and leaves the histogram zeroed
template <int PASS>
__global__ void __launch_bounds__(FIT_K * 32) k_fit_finish(FitInput in, const double* __restrict__ partial,
                                                           unsigned* __restrict__ hist, FitState* __restrict__ st,
                                                           gls_raw_nlf* __restrict__ out) {
    __shared__ double tot[FIT_K];
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    if (PASS > 0) {
        double v[(FIT_BLOCKS + 31) / 32];
#pragma unroll
        for (int j = 0; j < (FIT_BLOCKS + 31) / 32; j++) {  // every load issued before the sums
            const int b = lane + 32 * j;
            v[j] = b < FIT_BLOCKS ? partial[size_t(b) * FIT_K + k] : 0.0;
        }
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < (FIT_BLOCKS + 31) / 32; j++) t += v[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) tot[k] = t;
    } else if (threadIdx.x < 6) {
        tot[threadIdx.x] = double(hist[threadIdx.x]);
        hist[threadIdx.x] = 0;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const int n = nch(in);
    if (PASS == 0) {  // the variance bound from the class histogram (raw_converter.cpp:364-369)
        const double* h = tot;
        const double b = h[0] > 1e3 ? 1.0e-5 : h[1] > 1e3 ? 1.0e-4 : h[2] > 1e3 ? 1.0e-3
                       : h[3] > 1e3 ? 1.0e-2 : h[4] > 1e3 ? 1.0e-1 : 1.0;
        for (int c = 0; c < 4; c++) st->bound[c] = b;
    } else if (PASS == 1) {
        const double N = tot[16];
        for (int c = 0; c < n; c++) {
            const double sx = tot[c], sy = tot[4 + c], sxx = tot[8 + c], sxy = tot[12 + c];
            st->B[c] = max_s((N * sxy - sx * sy) / (N * sxx - sx * sx), 1e-8);
            st->A[c] = max_s((sy - st->B[c] * sx) / N, 1e-8);
        }
        st->N1 = N;
    } else if (PASS == 2) {
        for (int c = 0; c < n; c++) {
            st->err2[c] = tot[c] / st->N1;
            st->bound[c] = st->B[c];  // the second pass keeps variances under the fitted slope
        }
    } else {
        const double N = tot[16];
        double newErr2[4];
        bool better = true, nan = false;
        for (int c = 0; c < n; c++) {
            newErr2[c] = tot[17 + c] / N;
            nan = nan || isnan(newErr2[c]);
            better = better && (in.raw ? newErr2[c] < st->err2[c] : newErr2[c] <= st->err2[c]);
        }
        const bool accept = in.raw ? (N > 0.001 * in.pixels && !nan && better) : (better && N / in.pixels > 0.01);
        double A[4], B[4];
        for (int c = 0; c < n; c++) {
            A[c] = st->A[c];
            B[c] = st->B[c];
            if (accept) {
                const double sx = tot[c], sy = tot[4 + c], sxx = tot[8 + c], sxy = tot[12 + c];
                B[c] = max_s((N * sxy - sx * sy) / (N * sxx - sx * sx), 1e-8);
                A[c] = max_s((sy - B[c] * sx) / N, 1e-8);
            }
        }
        const double adj = double(__fmul_rn(in.exposure, in.exposure));  // a float product, as in the reference
        for (int c = 0; c < 4; c++) {
            out->a[c] = c < n ? float(A[c] * adj) : 0.f;
            out->b[c] = c < n ? float(B[c] * adj) : 0.f;
        }
    }
}

struct FitScratch {
    double* partial;
    FitState* st;
    unsigned* hist;
};

FitScratch fit_scratch(void* scratch) {
    char* p = static_cast<char*>(scratch);
    FitScratch f;
    f.partial = reinterpret_cast<double*>(p);
    p += size_t(FIT_BLOCKS) * FIT_K * sizeof(double);
    f.st = reinterpret_cast<FitState*>(p);
    p += sizeof(FitState);
    f.hist = reinterpret_cast<unsigned*>(p);
    return f;
}

template <bool RAW>
void launch_fit(const FitInput& in, const FitScratch& f, gls_raw_nlf* out, cudaStream_t s) {
    k_fit_finish<0><<<1, FIT_K * 32, 0, s>>>(in, f.partial, f.hist, f.st, out);
    k_fit_pass<1, RAW><<<FIT_BLOCKS, FIT_THREADS, 0, s>>>(in, f.st, f.partial);
    k_fit_finish<1><<<1, FIT_K * 32, 0, s>>>(in, f.partial, f.hist, f.st, out);
    k_fit_pass<2, RAW><<<FIT_BLOCKS, FIT_THREADS, 0, s>>>(in, f.st, f.partial);
    k_fit_finish<2><<<1, FIT_K * 32, 0, s>>>(in, f.partial, f.hist, f.st, out);
    k_fit_pass<3, RAW><<<FIT_BLOCKS, FIT_THREADS, 0, s>>>(in, f.st, f.partial);
    k_fit_finish<3><<<1, FIT_K * 32, 0, s>>>(in, f.partial, f.hist, f.st, out);
}

}  // namespace

// partial sums, the fit state and the class histogram (which each
// measurement leaves zeroed; zero the scratch when it is allocated)
size_t nlf_scratch_bytes() {
    return size_t(FIT_BLOCKS) * FIT_K * sizeof(double) + sizeof(FitState) + 8 * sizeof(unsigned);
}

template <class S>
int launch_measure_raw_nlf(Plane<S, 1> scaled, int pattern, Plane<float, 4> mean, Plane<float, 4> var,
                           float exposure, void* scratch, gls_raw_nlf* out, cudaStream_t s) {
    const FitScratch f = fit_scratch(scratch);
    const dim3 g((mean.w + RS_TX - 1) / RS_TX, (mean.h + RS_TY - 1) / RS_TY);
    const dim3 b(RS_TX, RS_TY);
    switch (pattern) {
        case 0: k_raw_stats<S, 0><<<g, b, 0, s>>>(scaled, mean, var, f.hist); break;
        case 1: k_raw_stats<S, 1><<<g, b, 0, s>>>(scaled, mean, var, f.hist); break;
        case 2: k_raw_stats<S, 2><<<g, b, 0, s>>>(scaled, mean, var, f.hist); break;
        default: k_raw_stats<S, 3><<<g, b, 0, s>>>(scaled, mean, var, f.hist); break;
    }
    FitInput in{reinterpret_cast<const float4*>(mean.p), reinterpret_cast<const float4*>(var.p), mean.w, mean.h,
                mean.pitch / 4, 1, double(scaled.w) * double(scaled.h), exposure};
    launch_fit<true>(in, f, out, s);
    return 8;
}

template <class S>
int launch_measure_ycc_nlf(Plane<S, 4> img, Plane<float, 4> stats, float exposure, void* scratch,
                           gls_raw_nlf* out, cudaStream_t s) {
    const FitScratch f = fit_scratch(scratch);
    auto run = [&](auto positions) {
        constexpr int P = decltype(positions)::value;
        const dim3 g((img.w + YS_TX - 1) / YS_TX, (img.h + YS_TY * P - 1) / (YS_TY * P));
        k_ycc_stats<S, P><<<g, dim3(YS_TX, YS_TY), 0, s>>>(img, stats, f.hist);
    };
    // four positions a thread, or two, where that leaves three blocks for each
    // of the 148 SMs. us with 1, 2, 4: 256x192 (192 tiles of 32 x 8) 4.8 5.8 8.0,
    // 400x300 (494) 6.2 6.6 7.9, 640x480 (1200) 10.0 8.9 10.1, 800x600 (1875)
    // 13.6 11.9 11.8, 2016x1512 65 45 40.
    const int tiles = ((img.w + YS_TX - 1) / YS_TX) * ((img.h + YS_TY - 1) / YS_TY);
    if (tiles >= 4 * 444) run(std::integral_constant<int, 4>{});
    else if (tiles >= 2 * 444) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 1>{});
    FitInput in{reinterpret_cast<const float4*>(stats.p), nullptr, stats.w, stats.h, stats.pitch / 4, 0,
                double(img.w) * double(img.h), exposure};
    launch_fit<false>(in, f, out, s);
    return 8;
}

template int launch_measure_raw_nlf<float>(Plane<float, 1>, int, Plane<float, 4>, Plane<float, 4>, float, void*,
                                           gls_raw_nlf*, cudaStream_t);
template int launch_measure_raw_nlf<__half>(Plane<__half, 1>, int, Plane<float, 4>, Plane<float, 4>, float, void*,
                                            gls_raw_nlf*, cudaStream_t);
template int launch_measure_ycc_nlf<float>(Plane<float, 4>, Plane<float, 4>, float, void*, gls_raw_nlf*,
                                           cudaStream_t);
template int launch_measure_ycc_nlf<__half>(Plane<__half, 4>, Plane<float, 4>, float, void*, gls_raw_nlf*,
                                            cudaStream_t);

}  // namespace gls
