// gls_pyramid.cu — kernels of PyramidProcessor<levels>::denoise
// (pyramid_processor.cpp:96-172): Gaussian-pyramid downsample, the
// reconstruct (noise subtraction) step, the per-level PCA patch basis
// (covariance + FP64 tridiagonal eigen-solve on the device; two-sided
// Jacobi on the host for GLS_HOST_PCA) and the 5x5-patch
// PCA projection. The block-matching denoise is in gls_blockmatch.cu.
#include <cmath>
#include <cstdio>

#include "gls_common.cuh"
#include "gls_kernels.h"
#include "gls_pca_pairs.h"
#include "gls_pyramid_dev.cuh"

namespace gls {

// --------------------------------------------------------------------------
// downsampleImageXYZ / downsampleImageXY, demosaic.metal:886-920: mean of
// four bilinear samples at texel-space (x*r - 0.5, (x+1)*r - 0.5) with
// r = in/out size (a 4x4 box for an exact halving). Positions are formed
// with explicit FP32 roundings, matching the oracle's FP32 run.
template <class S, int C>
__device__ __forceinline__ void downsample_px(const Plane<S, C>& in, const Plane<S, C>& out, float rx, float ry,
                                              int x, int y) {
    const float u[2] = {__fsub_rn(__fmul_rn(float(x), rx), 0.5f), __fsub_rn(__fmul_rn(float(x + 1), rx), 0.5f)};
    const float v[2] = {__fsub_rn(__fmul_rn(float(y), ry), 0.5f), __fsub_rn(__fmul_rn(float(y + 1), ry), 0.5f)};
    float acc[C > 2 ? 3 : 2] = {};
    constexpr int NC = C > 2 ? 3 : 2;
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const float fu = floorf(u[a]), fv = floorf(v[b]);
            const int xi = int(fu), yi = int(fv);
            const float ax = u[a] - fu, ay = v[b] - fv;
            float t00[4], t01[4], t10[4], t11[4];
            auto ld = [&](int xx, int yy, float* dst) {
                const S* p = in.pxc(xx, yy);
                if constexpr (C == 4) {
                    const f4 q = ld4<S>(p);
                    dst[0] = q.x; dst[1] = q.y; dst[2] = q.z;
                } else {
                    const f2 q = ld2<S>(p);
                    dst[0] = q.x; dst[1] = q.y;
                }
            };
            ld(xi, yi, t00);
            ld(xi + 1, yi, t01);
            ld(xi, yi + 1, t10);
            ld(xi + 1, yi + 1, t11);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const float top = t00[c] + (t01[c] - t00[c]) * ax;
                const float bot = t10[c] + (t11[c] - t10[c]) * ax;
                acc[c] += top + (bot - top) * ay;
            }
        }
    if constexpr (C == 4) {
        st4<S>(out.px(x, y), f4{0.25f * acc[0], 0.25f * acc[1], 0.25f * acc[2], 0.f});
    } else {
        st2<S>(out.px(x, y), f2{0.25f * acc[0], 0.25f * acc[1]});
    }
}

// The image and the gradient of a pyramid level in one launch (same sizes,
// same sample positions): PyramidProcessor::denoise's two downsamples
// (pyramid_processor.cpp:109-110).
template <class S>
__global__ void __launch_bounds__(256) k_downsample_pair(Plane<S, 4> img, Plane<S, 4> img_out, Plane<S, 2> grad,
                                                         Plane<S, 2> grad_out, float rx, float ry) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= img_out.w || y >= img_out.h) return;
    downsample_px<S, 4>(img, img_out, rx, ry, x, y);
    downsample_px<S, 2>(grad, grad_out, rx, ry, x, y);
}

template <class S>
__global__ void __launch_bounds__(256) k_subtract_noise(Plane<S, 4> in, Plane<S, 4> coarse, Plane<S, 4> coarse_den,
                                                        Plane<S, 2> grad, Plane<S, 4> out, SubtractArgs a, float rx,
                                                        float ry) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= in.w || y >= in.h) return;
    subtract_noise_px<S>(in, coarse, coarse_den, grad, out, a, rx, ry, x, y);
}

template <class S>
__global__ void __launch_bounds__(352, 3) k_pca_cov(Plane<S, 4> img, double* __restrict__ part, int group, int n_chunks) {
    __shared__ CovSmem sm;
    const int c0 = blockIdx.x * group;
    pca_cov_row<S>(img, part + size_t(blockIdx.x) * kPcaAcc, c0, min(c0 + group, n_chunks), sm);
}

constexpr int EJ_THREADS = 384;  // the prologue's 700 partial sums in two rounds, 168 registers for the one-warp phases

__global__ void __launch_bounds__(EJ_THREADS) k_pca_eigen(const double* __restrict__ part, int n_blocks,
                                                         int n_patches, float* __restrict__ basis, int* status) {
    __shared__ EigenSmem sm;
    pca_eigen_block(part, n_blocks, n_patches, basis, status, sm);
}

// --------------------------------------------------------------------------
// pcaProjection, demosaic.metal:774-796: 5x5 luma patch times the 25x8
// basis -> 8 coefficients per pixel, summed tap by tap. Bound by issue (200
// FMAs a pixel) and 48 B of traffic: two vertically adjacent pixels a thread
// share a tap's basis row and the patches' common rows, from a staged 36 x 20
// luma region. 2048x1536 FP32: 60 us, 86 with clamped reads of the image for
// every tap.
constexpr int PP_W = 32, PP_H = 16;

__global__ void __launch_bounds__(PP_W* PP_H / 2) k_pca_project(Plane<float, 4> img, const float* __restrict__ basis,
                                                                Plane<float, 8> out) {
    __shared__ float4 b[25][2];
    __shared__ float luma[PP_H + 4][PP_W + 4];
    const int tid = threadIdx.y * PP_W + threadIdx.x;
    const int x0 = blockIdx.x * PP_W, y0 = blockIdx.y * PP_H;
    if (tid < 200) reinterpret_cast<float*>(b)[tid] = basis[tid];
    for (int k = tid; k < (PP_H + 4) * (PP_W + 4); k += PP_W * PP_H / 2)
        luma[k / (PP_W + 4)][k % (PP_W + 4)] = *img.pxc(x0 - 2 + k % (PP_W + 4), y0 - 2 + k / (PP_W + 4));
    __syncthreads();
    const int x = x0 + threadIdx.x, yt = 2 * threadIdx.y, y = y0 + yt;
    if (x >= img.w) return;
    float acc[2][8] = {};
#pragma unroll
    for (int r = 0; r < 6; r++)
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const float v = luma[yt + r][threadIdx.x + i];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                if (r - p < 0 || r - p > 4) continue;
                const float4 u = b[(r - p) * 5 + i][0], w = b[(r - p) * 5 + i][1];
                const float row[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
#pragma unroll
                for (int c = 0; c < 8; c++) acc[p][c] = fmaf(row[c], v, acc[p][c]);
            }
        }
#pragma unroll
    for (int p = 0; p < 2; p++) {
        if (y + p >= img.h) break;
        float4* o = reinterpret_cast<float4*>(out.px(x, y + p));
        o[0] = make_float4(acc[p][0], acc[p][1], acc[p][2], acc[p][3]);
        o[1] = make_float4(acc[p][4], acc[p][5], acc[p][6], acc[p][7]);
    }
}

// ------------------------------------------------------------------ launchers
static inline dim3 grid2(int w, int h, dim3 b) { return dim3((w + b.x - 1) / b.x, (h + b.y - 1) / b.y); }

template <class S>
void launch_downsample_pair(Plane<S, 4> img, Plane<S, 4> img_out, Plane<S, 2> grad, Plane<S, 2> grad_out,
                            cudaStream_t s) {
    dim3 b(32, 8);
    k_downsample_pair<S><<<grid2(img_out.w, img_out.h, b), b, 0, s>>>(
        img, img_out, grad, grad_out, float(img.w) / float(img_out.w), float(img.h) / float(img_out.h));
}

template <class S>
void launch_subtract_noise(Plane<S, 4> in, Plane<S, 4> coarse, Plane<S, 4> coarse_den, Plane<S, 2> grad,
                           Plane<S, 4> out, const SubtractArgs& a, cudaStream_t s) {
    dim3 b(32, 8);
    k_subtract_noise<S><<<grid2(in.w, in.h, b), b, 0, s>>>(in, coarse, coarse_den, grad, out, a,
                                                          float(coarse.w) / float(in.w), float(coarse.h) / float(in.h));
}

int pca_cov_chunks(int w, int h) {
    const int n = (w / 8) * (h / 8);
    return n <= 0 ? 0 : (n + PC_CHUNK - 1) / PC_CHUNK;
}

int pca_cov_rows(int w, int h) {
    const int chunks = pca_cov_chunks(w, h), g = pca_cov_group(chunks);
    return (chunks + g - 1) / g;
}

template <class S>
void launch_pca_cov(Plane<S, 4> img, double* part, cudaStream_t s) {
    const int rows = pca_cov_rows(img.w, img.h);
    if (rows == 0) return;
    const int chunks = pca_cov_chunks(img.w, img.h);
    k_pca_cov<S><<<rows, 352, 0, s>>>(img, part, pca_cov_group(chunks), chunks);
}

template <class S>
void launch_pca_cov_rows(Plane<S, 4> img, double* part, int rows, cudaStream_t s) {
    if (rows > 0) k_pca_cov<S><<<rows, 352, 0, s>>>(img, part, 1, pca_cov_chunks(img.w, img.h));
}
template void launch_pca_cov_rows<float>(Plane<float, 4>, double*, int, cudaStream_t);
template void launch_pca_cov_rows<__half>(Plane<__half, 4>, double*, int, cudaStream_t);

void launch_pca_eigen(const double* part, int n_blocks, int n_patches, float* basis, int* status, cudaStream_t s) {
    k_pca_eigen<<<1, EJ_THREADS, 0, s>>>(part, n_blocks, n_patches, basis, status);
}

void launch_pca_project(Plane<float, 4> img, const float* basis, Plane<float, 8> out, cudaStream_t s) {
    k_pca_project<<<grid2(img.w, img.h, dim3(PP_W, PP_H)), dim3(PP_W, PP_H / 2), 0, s>>>(img, basis, out);
}

// Host FP64 eigen-solve of the same accumulators: the per-level host PCA of
// the reference (pyramid_processor.cpp:148-149), for the GLS_HOST_PCA path.
void host_pca_basis(const double* part, int n_blocks, int n_patches, float* basis) {
    double acc[kPcaAcc];
    for (int t = 0; t < kPcaAcc; t++) {
        double v = 0.0;
        for (int b = 0; b < n_blocks; b++) v += part[b * kPcaAcc + t];
        acc[t] = v;
    }
    if (n_patches < 2) {
        for (int t = 0; t < 200; t++) basis[t] = ((t / 8) == (t % 8)) ? 1.f : 0.f;
        return;
    }
    double A[25][25], V[25][25];
    const double n = double(n_patches);
    for (int i = 0; i < 25; i++)
        for (int j = 0; j < 25; j++) {
            const int r = std::min(i, j), c = std::max(i, j);
            const int idx = pca_tri_index(r, c);
            A[i][j] = (acc[idx] - n * (acc[325 + i] / n) * (acc[325 + j] / n)) / (n - 1.0);
            V[i][j] = i == j ? 1.0 : 0.0;
        }
    for (int sweep = 0; sweep < 100; sweep++) {
        double off = 0, tot = 0;
        for (int i = 0; i < 25; i++)
            for (int j = 0; j < 25; j++) {
                tot += A[i][j] * A[i][j];
                if (i != j) off += A[i][j] * A[i][j];
            }
        if (off <= 1e-26 * tot || off == 0) break;
        for (int p = 0; p < 24; p++)
            for (int q = p + 1; q < 25; q++) {
                const double apq = A[p][q];
                if (std::fabs(apq) < 1e-300) continue;
                const double theta = (A[q][q] - A[p][p]) / (2 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1));
                const double c = 1 / std::sqrt(t * t + 1), s = t * c;
                for (int k = 0; k < 25; k++) {
                    const double akp = A[k][p], akq = A[k][q];
                    A[k][p] = c * akp - s * akq;
                    A[k][q] = s * akp + c * akq;
                }
                for (int k = 0; k < 25; k++) {
                    const double apk = A[p][k], aqk = A[q][k];
                    A[p][k] = c * apk - s * aqk;
                    A[q][k] = s * apk + c * aqk;
                }
                for (int k = 0; k < 25; k++) {
                    const double vkp = V[k][p], vkq = V[k][q];
                    V[k][p] = c * vkp - s * vkq;
                    V[k][q] = s * vkp + c * vkq;
                }
            }
    }
    int order[25];
    for (int k = 0; k < 25; k++) order[k] = k;
    for (int k = 1; k < 25; k++) {
        const int e = order[k];
        int m = k - 1;
        while (m >= 0 && A[order[m]][order[m]] < A[e][e]) {
            order[m + 1] = order[m];
            m--;
        }
        order[m + 1] = e;
    }
    double ev[25], evec[25 * 25], work[200];
    for (int c = 0; c < 25; c++) {
        ev[c] = A[order[c]][order[c]];
        for (int r = 0; r < 25; r++) evec[r * 25 + c] = V[r][order[c]];
    }
    select_pca_basis(ev, evec, 25, work, basis);
}

#define GLS_INST(S)                                                                                              \
    template void launch_downsample_pair<S>(Plane<S, 4>, Plane<S, 4>, Plane<S, 2>, Plane<S, 2>, cudaStream_t);  \
    template void launch_subtract_noise<S>(Plane<S, 4>, Plane<S, 4>, Plane<S, 4>, Plane<S, 2>, Plane<S, 4>,     \
                                           const SubtractArgs&, cudaStream_t);                                   \
    template void launch_pca_cov<S>(Plane<S, 4>, double*, cudaStream_t);
GLS_INST(float)
GLS_INST(__half)
#undef GLS_INST

}  // namespace gls
