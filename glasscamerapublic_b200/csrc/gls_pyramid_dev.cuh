// gls_pyramid_dev.cuh — device code of one pyramid level shared by the
// stream kernels (gls_pyramid.cu) and the persistent batch kernel
// (gls_blockmatch.cu): a pixel of the reconstruct step, a covariance
// partial row, and the eigen-solve of the level's PCA basis. Both callers
// run the same code, so their results are bit-identical.
#pragma once

#include "gls_common.cuh"
#include "gls_kernels.h"
#include "gls_pca_pairs.h"

namespace gls {

// --------------------------------------------------------------------------
// subtractNoiseImage, demosaic.metal:922-959: subtract the coarse level's
// removed noise (bilinear up-sampled) and apply the noise-gated sharpening.
template <class S>
__device__ __forceinline__ void bilin3(const Plane<S, 4>& p, float u, float v, float out[3]) {
    const float fu = floorf(u), fv = floorf(v);
    const int xi = int(fu), yi = int(fv);
    const float ax = u - fu, ay = v - fv;
    const f4 a = ld4<S>(p.pxc(xi, yi)), b = ld4<S>(p.pxc(xi + 1, yi));
    const f4 c = ld4<S>(p.pxc(xi, yi + 1)), d = ld4<S>(p.pxc(xi + 1, yi + 1));
    const float av[3] = {a.x, a.y, a.z}, bv[3] = {b.x, b.y, b.z}, cv[3] = {c.x, c.y, c.z}, dv[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float top = av[k] + (bv[k] - av[k]) * ax;
        const float bot = cv[k] + (dv[k] - cv[k]) * ax;
        out[k] = top + (bot - top) * ay;
    }
}

// One pixel of subtractNoiseImage (demosaic.metal:922-959): the layer at
// (x, y) from the level's image, the coarse level's noisy and denoised
// images (bilinear, texel position ((x + 0.5) r - 0.5)) and the gradient.
template <class S>
__device__ __forceinline__ void subtract_noise_px(const Plane<S, 4>& in, const Plane<S, 4>& coarse,
                                                  const Plane<S, 4>& coarse_den, const Plane<S, 2>& grad,
                                                  const Plane<S, 4>& out, const SubtractArgs& a, float rx, float ry,
                                                  int x, int y) {
    const float u = __fsub_rn(__fmul_rn(__fadd_rn(float(x), 0.5f), rx), 0.5f);
    const float v = __fsub_rn(__fmul_rn(__fadd_rn(float(y), 0.5f), ry), 0.5f);
    const f4 ip = ld4<S>(in.px(x, y));
    float p1[3], pd[3];
    bilin3(coarse, u, v, p1);
    bilin3(coarse_den, u, v, pd);
    const float ipv[3] = {ip.x, ip.y, ip.z};
    float dn[3];
#pragma unroll
    for (int c = 0; c < 3; c++) dn[c] = ipv[c] - (c == 0 ? a.luma_weight : 1.f) * (p1[c] - pd[c]);
    float alpha = a.sharpening;
    if (a.sharpening > 1.f) {
        const f2 g = ld2<S>(grad.px(x, y));
        const float gm = sqrtf(g.x * g.x + g.y * g.y);
        const float sigma = sqrtf(a.nlf_a + a.nlf_b * pd[0]);
        const float detail = smoothstepf(sigma, 4.f * sigma, gm) * (1.f - smoothstepf(0.75f, 0.95f, pd[0])) *
                             smoothstepf(0.05f, 0.1f, pd[0]);
        alpha = 1.f + (alpha - 1.f) * detail;
    }
    f4 o;
    o.x = fmaxf(mixf(pd[0], dn[0], alpha), 0.f);
    o.y = mixf(pd[1], dn[1], alpha);
    o.z = mixf(pd[2], dn[2], alpha);
    o.w = ip.w;
    st4<S>(out.px(x, y), o);
}

// --------------------------------------------------------------------------
// PCA patch covariance: collectPatches (demosaic.metal:755-772) fused with
// the covariance reduction of build_pca_space (PCA.cpp:29-33). Patches are
// the 5x5 luma neighbourhoods of (8x, 8y), x < W/8, y < H/8, taken in
// chunks of 64. Partial row r holds the FP64 sums over chunks
// [g r, g (r + 1)) (g chunks per row): the upper triangle of sum p p^T
// (325, indexed by pca_tri_index) then sum p (25). A block stages a
// chunk at a time in shared memory, converted to FP64 once per value; a
// thread issues all of its loads of a round before it stores any (the
// rounds are latency-bound: a few loads per thread, from L2). Its threads
// own the 350 accumulators (thread t the ones t, t + blockDim, ...), each
// summed patch by patch in four partial sums (patch k of the row into sum
// k mod 4), so a row's bits do not depend on the block size or the
// staging. The rows are summed in order by the eigen-solve, so the result
// does not depend on scheduling (no atomics).
constexpr int PC_CHUNK = kPcaChunk;
constexpr int PC_STAGE = PC_CHUNK;                           // patches staged per round
constexpr int PC_LOADS = (PC_STAGE * kPcaDim + 255) / 256;   // loads in flight per thread (256+ threads)

struct CovSmem {
    double sp[PC_STAGE][kPcaDim + 1];
};

template <class S>
__device__ __forceinline__ void pca_cov_row(Plane<S, 4> img, double* __restrict__ row, int chunk0, int chunk1,
                                            CovSmem& sm) {
    const int gw = img.w / 8, gh = img.h / 8;
    const int n = gw * gh;
    const int t = threadIdx.x, nth = blockDim.x;
    // four partial sums per accumulator (patches k = 0, 1, 2, 3 mod 4): FP64
    // chains a quarter as long; added in a fixed order at the end
    double sum[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
    int r[2] = {0, 0}, c[2] = {-1, -1};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int a = t + j * nth;
        if (a < kPcaTri) pca_pair(a, r[j], c[j]);
        else if (a < kPcaAcc) r[j] = a - kPcaTri;
    }
    // patch index -> (column, row) of the patch grid by a multiply-high:
    // q = umulhi(p, floor((2^32 - 1) / gw) + 1) is p / gw exactly while
    // p * gw < 2^32 (every frame up to ~100 MP); a division otherwise
    const bool fast_div = gw > 1 && uint64_t(n) * uint64_t(gw) < (1ull << 32);
    const uint32_t gmul = fast_div ? 0xffffffffu / uint32_t(gw) + 1u : 0u;
    const int p_end = min(chunk1 * PC_CHUNK, n);
    for (int base = chunk0 * PC_CHUNK; base < p_end; base += PC_STAGE) {
        const int cnt = min(PC_STAGE, p_end - base);
        const int nv = cnt * kPcaDim;
        for (int i0 = 0; i0 < nv; i0 += PC_LOADS * nth) {
            float v[PC_LOADS];
#pragma unroll
            for (int u = 0; u < PC_LOADS; u++) {
                const int i = i0 + t + u * nth;
                v[u] = 0.f;
                if (i < nv) {
                    const int k = i / kPcaDim, e = i - k * kPcaDim;  // constant divisors
                    const int pidx = base + k;
                    const int prow = fast_div ? int(__umulhi(uint32_t(pidx), gmul)) : pidx / gw;
                    const int ey = e / 5;
                    const int px = (pidx - prow * gw) * 8 + (e - ey * 5) - 2, py = prow * 8 + ey - 2;
                    v[u] = to_f(*img.pxc(px, py));
                }
            }
#pragma unroll
            for (int u = 0; u < PC_LOADS; u++) {
                const int i = i0 + t + u * nth;
                if (i < nv) sm.sp[i / kPcaDim][i % kPcaDim] = double(v[u]);
            }
        }
        __syncthreads();
        // patch k into partial sum k mod 4 (base is a multiple of 4, and cnt
        // is but in the last round of the level): products by FMA, the 25
        // component sums by additions
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int a = t + j * nth;
            if (a >= kPcaAcc) continue;
            const int rr = r[j], cc = c[j];
            double* s4 = sum[j];
            int k = 0;
            if (a < kPcaTri) {
                for (; k + 4 <= cnt; k += 4) {
#pragma unroll
                    for (int q = 0; q < 4; q++) s4[q] = fma(sm.sp[k + q][rr], sm.sp[k + q][cc], s4[q]);
                }
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (k + q < cnt) s4[q] = fma(sm.sp[k + q][rr], sm.sp[k + q][cc], s4[q]);
            } else {
                for (; k + 4 <= cnt; k += 4) {
#pragma unroll
                    for (int q = 0; q < 4; q++) s4[q] += sm.sp[k + q][rr];
                }
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (k + q < cnt) s4[q] += sm.sp[k + q][rr];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int a = t + j * nth;
        if (a < kPcaAcc) row[a] = ((sum[j][0] + sum[j][1]) + sum[j][2]) + sum[j][3];
    }
}

// --------------------------------------------------------------------------
// Symmetric eigen-solve of the 25x25 patch covariance (replaces Eigen's
// SelfAdjointEigenSolver, PCA.cpp:36), FP64, one block. Only the 8 largest
// eigenpairs are needed, so the solve is the tridiagonal route of Golub &
// Van Loan (Matrix Computations, 4th ed.): section 8.3.1 and the
// bisection / inverse-iteration methods of sections 8.4.1 and 8.2.2
// (the tred2 / tridiagonal bisection / tinvit sequence of EISPACK):
//   1. Householder tridiagonalisation, A = Q T Q^T, Q = H_0 ... H_22, by
//      seven warps, the matrix in shared memory: eight lanes to a row form
//      its sums (three terms a lane, three shuffles), every row for itself, and
//      update it; three barriers a step;
//   2. the 8 largest eigenvalues of T by Sturm-sequence multisection:
//      warp w brackets eigenvalue 24 - w (ascending order); its 32 lanes
//      count the eigenvalues below 32 points of the bracket, which shrinks
//      33-fold per round (9 rounds: 2e-14 of the spectrum width). The counts
//      are the sign changes of the leading principal minors' recurrence on T
//      scaled by a power of two, one FMA a term on the serial path; a
//      recurrence that ends at zero is counted by its pivots;
//   3. the eigenvectors of T by inverse iteration, lane c of one warp for
//      eigenvector c: T - lambda I is factored once with partial pivoting by
//      selects (no divergence) and solved twice from a start vector of its
//      own; tiny pivots are raised to eps ||T|| so the solve stays finite;
//   4. the back-transform z = H_0 (H_1 (... H_22 y)) in the same lanes, the
//      vector in registers, the reflectors read by broadcast;
//   5. Gram-Schmidt (modified, twice) of the 8 vectors in eigenvalue order if
//      two eigenvalues lie close together (exactly equal ones give an
//      orthonormal basis of their eigenspace; distinct ones are orthogonal
//      already).
// The top-8 eigenvectors (descending eigenvalue, each signed so its
// largest-magnitude entry is positive; eigenvalues <= 1e-9 of the largest
// completed as in select_pca_basis) are written as a row-major 25x8 FP32
// basis. Every reduction has a fixed order, so the result is deterministic.
// status receives the number of inverse-iteration solves per vector (2), or
// -1 when a vector came out non-finite (the basis is then still written). The
// eigenvalues of a T that is not finite, or too small to scale, count as 0: the
// basis is select_pca_basis's unit vectors.
// Bound by the serial chain on one SM: 29 us (tridiagonalisation 14, Sturm 4.5,
// inverse iteration to the basis 6, the launch and the row sums 4), 68 us with
// block-wide phases for every step and the pivot form of the Sturm sequence.
// Matrix rows in registers (one warp with a row per lane; eight lanes with
// two barriers a step) were no faster: 22 and 16 us for the tridiagonalisation.
constexpr int EJ_N = 25, EJ_TOP = 8, EJ_INV_ITERS = 2, EJ_MSEC_ROUNDS = 9;
constexpr int EJ_HH = 224;  // threads of the tridiagonalisation: eight to a row

// 1 / x to FP64 accuracy: the hardware approximation refined by two
// Newton-Raphson steps r <- r + r (1 - x r), each doubling the correct bits.
__device__ __forceinline__ double rcp_nr(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

// 1 / sqrt(x) to FP64 accuracy for normal x > 0: the hardware approximation
// refined by two steps of Newton's method on f(r) = 1 / r^2 - x,
// r <- r (3 - x r^2) / 2, each doubling the correct bits.
__device__ __forceinline__ double rsqrt_nr(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double hx = 0.5 * x;
    r = r * fma(-hx * r, r, 1.5);
    return r * fma(-hx * r, r, 1.5);
}

// Number of eigenvalues of the symmetric tridiagonal (d, e) below x: the
// signs of the pivots of T - x I (Sturm sequence); a pivot smaller than
// pivmin in magnitude is replaced by -pivmin.
static __device__ __noinline__ int sturm_count_pivots(const double* d, const double* ee, double x, double pivmin) {
    double q = d[0] - x;
    if (fabs(q) < pivmin) q = -pivmin;
    int cnt = q < 0.0;
#pragma unroll 1
    for (int i = 1; i < EJ_N; i++) {
        q = fma(-ee[i - 1], rcp_nr(q), d[i] - x);
        if (fabs(q) < pivmin) q = -pivmin;
        cnt += q < 0.0;
    }
    return cnt;
}

// The same as the sign changes of the leading minors p_i of T - x I,
// p_i = (d_i - x) p_(i-1) - e_(i-1)^2 p_(i-2), for entries of T of at most 1 in
// size (24 factors below 4 cannot overflow; both terms are rescaled by a power
// of two every 8 steps against underflow). A zero minor between nonzero ones
// counts once whichever sign it is given; a sequence that has run to zero is
// counted by its pivots.
__device__ __forceinline__ int sturm_count(const double* d, const double* ee, double x, double pivmin) {
    double p0 = 1.0, p1 = d[0] - x;
    unsigned cnt = unsigned(__double2hiint(p1)) >> 31;  // sign bits: the FP64 pipe is the limit here
#pragma unroll 1  // a body of 8 steps stays in the instruction cache
    for (int i0 = 1; i0 < EJ_N; i0 += 8) {
#pragma unroll
        for (int i = i0; i < i0 + 8; i++) {
            const double p2 = fma(d[i] - x, p1, -(ee[i - 1] * p0));
            cnt += unsigned(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
            p0 = p1;
            p1 = p2;
        }
        const int ex = max(__double2hiint(p0) & 0x7fffffff, __double2hiint(p1) & 0x7fffffff) >> 20;  // biased exponent
        const double sc = __hiloint2double((2046 - min(ex, 2045)) << 20, 0);                        // 2^(1023 - ex)
        p0 *= sc;
        p1 *= sc;
    }
    return p1 != 0.0 ? int(cnt) : sturm_count_pivots(d, ee, x, pivmin);
}

// sum_{j = 1..24} a[j] b[j] in four interleaved partial FP64 chains, added in
// a fixed order: a quarter of the latency of one chain
__device__ __forceinline__ double dot24(const double (&a)[EJ_N], const double (&b)[EJ_N]) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 1; j < EJ_N; j++) s[j & 3] = fma(a[j], b[j], s[j & 3]);
    return (s[1] + s[2]) + (s[3] + s[0]);
}

// the 25 values of a 16-byte aligned shared vector
__device__ __forceinline__ void load25(const double* p, double (&v)[EJ_N]) {
#pragma unroll
    for (int j = 0; j < EJ_N - 1; j += 2) {
        const double2 t = *reinterpret_cast<const double2*>(p + j);
        v[j] = t.x;
        v[j + 1] = t.y;
    }
    v[EJ_N - 1] = p[EJ_N - 1];
}

struct EigenSmem {
    alignas(16) double V[EJ_N - 2][EJ_N + 1];  // Householder vectors (zero above k + 1)
    double ax[EJ_N], w[EJ_N];                  // a tridiagonalisation step's vectors
    alignas(16) double q[EJ_N + 1];            // the vector that Gram-Schmidt broadcasts
    double A[EJ_N][EJ_N + 1];                  // covariance
    double beta[EJ_N - 2];
    double d[EJ_N], e[EJ_N], ee[EJ_N];
    double lam[EJ_TOP], tnorm;
    // inverse iteration, lane c for eigenvector c: the pivoted LU of T - lambda I
    double ru0[EJ_N][EJ_TOP], u1[EJ_N][EJ_TOP], u2[EJ_N][EJ_TOP], l[EJ_N][EJ_TOP];
    unsigned char piv[EJ_N][EJ_TOP];
    double Z[EJ_N][EJ_TOP + 1];                // eigenvectors of A, column c = the c-th largest
    double work[200];
    double acc[kPcaAcc], part1[kPcaAcc], part2[kPcaAcc];
    int bad;
};

// The solve by one block of at least 8 warps (any size: every loop strides
// by the block size, and the bits do not depend on it).
__device__ inline void pca_eigen_block(const double* __restrict__ part, int n_blocks, int n_patches,
                                float* __restrict__ basis, int* status, EigenSmem& sm) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nth = blockDim.x;

    if (n_patches < 2) {
        for (int k = t; k < 25 * 8; k += nth) basis[k] = ((k / 8) == (k % 8)) ? 1.f : 0.f;
        if (t == 0 && status) *status = 0;
        return;
    }
    // ---- partial rows summed in a fixed order: two halves of the row range
    //      per accumulator, 32 loads in flight each, then added
    {
        const int half = (n_blocks + 1) / 2;
        for (int q = t; q < 2 * kPcaAcc; q += nth) {
            const int h = q / kPcaAcc, a = q % kPcaAcc;
            const int b0 = h == 0 ? 0 : half, b1 = h == 0 ? half : n_blocks;
            double v = 0.0;
            int b = b0;
            for (; b + 32 <= b1; b += 32) {  // 32 loads in flight
                double x[32];
#pragma unroll
                for (int k = 0; k < 32; k++) x[k] = part[size_t(b + k) * kPcaAcc + a];
#pragma unroll
                for (int k = 0; k < 32; k++) v += x[k];
            }
#pragma unroll 4
            for (; b < b1; b++) v += part[size_t(b) * kPcaAcc + a];
            (h == 0 ? sm.part1 : sm.part2)[a] = v;
        }
        if (t == 0) sm.bad = 0;
        __syncthreads();
        for (int a = t; a < kPcaAcc; a += nth) sm.acc[a] = sm.part1[a] + sm.part2[a];
    }
    __syncthreads();
    // ---- covariance from raw moments, (sum pp^T - n m m^T) / (n - 1)
    for (int k = t; k < EJ_N * EJ_N; k += nth) {
        const int i = k / EJ_N, j = k % EJ_N;
        const int idx = pca_tri_index(min(i, j), max(i, j));
        const double n = double(n_patches);
        const double mi = sm.acc[325 + i] / n, mj = sm.acc[325 + j] / n;
        sm.A[i][j] = (sm.acc[idx] - n * mi * mj) / (n - 1.0);
    }
    __syncthreads();

    // ---- 1. Householder tridiagonalisation, eight lanes to a row. With x
    //         column k below the diagonal, v = x - alpha e1, beta = 2 / v.v:
    //         p = beta A v = beta (A x - alpha A e1), and v.A v = x.A x -
    //         2 alpha (A x)_1 + alpha^2 A_11 (x.A e1 is (A x)_1), so A x and w are
    //         the only vectors exchanged; w = p - (beta / 2) (p.v) v, then
    //         A -= v w^T + w v^T on the trailing block.
    if (t < EJ_HH) {
        const int i = t >> 3, s8 = t & 7, row = min(i, EJ_N - 1);
        auto bar = [] { asm volatile("bar.sync 1, %0;" ::"n"(EJ_HH) : "memory"); };
        auto sum8 = [](double v) {  // over the row's eight lanes
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            return v + __shfl_xor_sync(0xffffffffu, v, 1);
        };
#pragma unroll 1
        for (int k = 0; k < EJ_N - 2; k++) {
            const bool below = i > k && i < EJ_N;
            double x[3], a[3];
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const int j = k + 1 + s8 + 8 * m;
                x[m] = j < EJ_N ? sm.A[j][k] : 0.0;
                a[m] = j < EJ_N ? sm.A[row][j] : 0.0;
            }
            const double x1 = sm.A[k + 1][k], xi = sm.A[row][k], ai1 = sm.A[row][k + 1], a11 = sm.A[k + 1][k + 1];
            const double n2 = sum8(fma(x[2], x[2], fma(x[1], x[1], x[0] * x[0])));
            const double ax = sum8(fma(a[2], x[2], fma(a[1], x[1], a[0] * x[0])));
            if (s8 == 0 && below) sm.ax[i] = ax;
            // the norm and 1 / (v.v / 2) by refined hardware approximations:
            // the IEEE square root and division are long serial sequences
            const bool skip = !(n2 > 1e-280);  // the column is already reduced
            const double nrm = skip ? 0.0 : n2 * rsqrt_nr(n2);
            const double alpha = x1 >= 0.0 ? -nrm : nrm;
            const double beta = skip ? 0.0 : rcp_nr(n2 - alpha * x1);  // v.v / 2 > 0 unless the column is zero
            const double v1 = skip ? 0.0 : x1 - alpha;
            bar();
            double xy = 0.0;
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const int j = k + 1 + s8 + 8 * m;
                if (j < EJ_N) xy = fma(x[m], sm.ax[j], xy);
            }
            const double vav = fma(alpha * alpha, a11, fma(-2.0 * alpha, sm.ax[k + 1], sum8(xy)));
            const double K = 0.5 * beta * beta * vav;  // (beta / 2) p.v
            const double v = skip || !below ? 0.0 : (i == k + 1 ? v1 : xi);
            const double w = skip || !below ? 0.0 : beta * (ax - alpha * ai1) - K * v;
            if (s8 == 0 && i < EJ_N) {
                sm.w[i] = w;
                sm.V[k][i] = v;
            }
            if (t == 0) {
                sm.beta[k] = beta;
                sm.d[k] = sm.A[k][k];
                sm.e[k] = skip ? x1 : alpha;
            }
            bar();
            if (below && !skip) {
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    const int j = k + 1 + s8 + 8 * m;
                    if (j < EJ_N) sm.A[i][j] = a[m] - fma(v, sm.w[j], w * (j == k + 1 ? v1 : x[m]));
                }
            }
            bar();
        }
    }
    if (warp == 0) {
        if (lane == 0) {
            sm.d[EJ_N - 2] = sm.A[EJ_N - 2][EJ_N - 2];
            sm.d[EJ_N - 1] = sm.A[EJ_N - 1][EJ_N - 1];
            sm.e[EJ_N - 2] = sm.A[EJ_N - 1][EJ_N - 2];
            sm.e[EJ_N - 1] = 0.0;
        }
        __syncwarp();
        // T scaled by a power of two to a Gershgorin bound in [1/2, 1): exact, and
        // neither the eigenvectors nor the rank threshold depend on it. Only the
        // bound's exponent is needed: the largest high word
        double b = 0.0;
        if (lane < EJ_N) b = fabs(sm.d[lane]) + fabs(sm.e[lane]) + (lane > 0 ? fabs(sm.e[lane - 1]) : 0.0);
        const unsigned ex = __reduce_max_sync(0xffffffffu, unsigned(__double2hiint(b))) >> 20;
        const double sc = ex > 64 && ex < 2000 ? __hiloint2double((2045 - ex) << 20, 0) : 1.0;
        if (lane < EJ_N) {
            const double e = sm.e[lane] * sc;
            sm.d[lane] *= sc;
            sm.ee[lane] = e * e;
            sm.e[lane] = e;
        }
        if (lane == 0) sm.tnorm = ex > 64 && ex < 2000 ? 1.0 : 0.0;  // 0: no eigenvalue to find
    }
    __syncthreads();

    // ---- 2. the 8 largest eigenvalues by Sturm multisection, warp w for
    //         eigenvalue index 24 - w (ascending)
    const double tnorm = sm.tnorm;
    if (warp < EJ_TOP) {
        double lo = -tnorm, hi = tnorm;
        constexpr double pivmin = 1e-290;
        const int m = EJ_N - 1 - warp;
#pragma unroll 1
        for (int r = 0; r < EJ_MSEC_ROUNDS; r++) {
            if (!(hi - lo > 4.4e-16 * fmax(fabs(lo), fabs(hi)) + pivmin)) break;  // warp-uniform
            const double x = lo + (hi - lo) * (double(lane + 1) * (1.0 / 33.0));
            const int c = sturm_count(sm.d, sm.ee, x, pivmin);
            const unsigned above = __ballot_sync(0xffffffffu, c > m);
            const int first = above ? __ffs(above) - 1 : 32;
            const double xl = __shfl_sync(0xffffffffu, x, max(first - 1, 0));
            const double xh = __shfl_sync(0xffffffffu, x, min(first, 31));
            if (first > 0) lo = xl;
            if (first < 32) hi = xh;
        }
        if (lane == 0) sm.lam[warp] = 0.5 * (lo + hi);
    }
    __syncthreads();
    if (warp != 0) return;

    // ---- 3. inverse iteration on T, lane c for eigenvector c
    const int c = min(lane, EJ_TOP - 1);
    double y[EJ_N];
    {
        const double lam = sm.lam[c];
        const double tiny = fmax(2.2e-16 * tnorm, 1e-290);
        // factor T - lam I = P L U (Gaussian elimination, partial pivoting);
        // U has the diagonal u0 (kept as 1 / u0) and two super-diagonals
        double a = sm.d[0] - lam, b = sm.e[0];
        if (lane < EJ_TOP) {
#pragma unroll 4
            for (int k = 0; k < EJ_N - 1; k++) {
                const double cl = sm.e[k];                 // sub-diagonal entry of row k + 1
                const double an = sm.d[k + 1] - lam;       // diagonal of row k + 1
                const double bn = sm.e[k + 1];             // 0 for the last row
                const bool swap = fabs(a) < fabs(cl);      // rows k and k + 1 interchanged
                double piv = swap ? cl : a;
                if (fabs(piv) < tiny) piv = piv < 0.0 ? -tiny : tiny;
                const double rp = rcp_nr(piv);
                const double mult = (swap ? a : cl) * rp;
                const double u1 = swap ? an : b, u2 = swap ? bn : 0.0;
                sm.ru0[k][c] = rp;
                sm.u1[k][c] = u1;
                sm.u2[k][c] = u2;
                sm.l[k][c] = mult;
                sm.piv[k][c] = swap;
                a = (swap ? b : an) - mult * u1;
                b = (swap ? 0.0 : bn) - mult * u2;
            }
            if (fabs(a) < tiny) a = a < 0.0 ? -tiny : tiny;
            sm.ru0[EJ_N - 1][c] = rcp_nr(a);
        }
        // start vector of its own per eigenvector (deterministic)
#pragma unroll
        for (int i = 0; i < EJ_N; i++) y[i] = 1.0 + (0.25 / 13.0) * double(((i + 1) * (7 + 4 * c)) % 13);
        __syncwarp();
#pragma unroll 1
        for (int it = 0; it < EJ_INV_ITERS; it++) {
#pragma unroll
            for (int k = 0; k < EJ_N - 1; k++) {           // apply P and L^-1
                const bool swap = sm.piv[k][c];
                const double up = swap ? y[k + 1] : y[k], dn = swap ? y[k] : y[k + 1];
                y[k] = up;
                y[k + 1] = dn - sm.l[k][c] * up;
            }
            y[EJ_N - 1] *= sm.ru0[EJ_N - 1][c];            // U^-1
            y[EJ_N - 2] = (y[EJ_N - 2] - sm.u1[EJ_N - 2][c] * y[EJ_N - 1]) * sm.ru0[EJ_N - 2][c];
#pragma unroll
            for (int k = EJ_N - 3; k >= 0; k--)
                y[k] = (fma(-sm.u2[k][c], y[k + 2], y[k]) - sm.u1[k][c] * y[k + 1]) * sm.ru0[k][c];
            double m[4] = {0.0, 0.0, 0.0, 0.0};            // rescale by the largest entry
#pragma unroll
            for (int i = 0; i < EJ_N; i++) m[i & 3] = fmax(m[i & 3], fabs(y[i]));
            const double mx = fmax(fmax(m[0], m[1]), fmax(m[2], m[3]));
            const double inv = mx > 1e-290 && mx < 1e300 ? rcp_nr(mx) : 0.0;
#pragma unroll
            for (int i = 0; i < EJ_N; i++) y[i] *= inv;
        }
    }
    // ---- 4. back-transform z = H_0 (H_1 (... H_22 y)), lane c for vector c
#pragma unroll 1
    for (int k = EJ_N - 3; k >= 0; k--) {
        double v[EJ_N];
        load25(sm.V[k], v);  // zero for entries <= k, all zero for a skipped column
        const double s = sm.beta[k] * dot24(v, y);
#pragma unroll
        for (int i = 1; i < EJ_N; i++) y[i] = fma(-s, v[i], y[i]);
    }
    // ---- 5. normalisation; a non-finite vector is zeroed. Vectors of
    //         eigenvalues 1e-7 of ||T|| apart are orthogonal to 2e-9 as they
    //         are (rounding over the gap, below FP32); closer ones go through
    //         Gram-Schmidt in eigenvalue order, vector g subtracted from the
    //         later ones, twice
    bool close = false;
#pragma unroll
    for (int k = 0; k + 1 < EJ_TOP; k++) close = close || !(sm.lam[k] - sm.lam[k + 1] > 1e-7);
    const int steps = close ? 2 * EJ_TOP : 0;
#pragma unroll 1
    for (int step = -1; step < steps; step++) {
        const int g = step < 0 ? -1 : step % EJ_TOP;
        if (step < 0 || lane == g) {  // the first round normalises every vector
            const double nn = fma(y[0], y[0], dot24(y, y));
            const bool ok = nn > 1e-290 && nn < 1e300;
            const double r = ok ? rsqrt_nr(nn) : 0.0;
            if (!ok) sm.bad = 1;
#pragma unroll
            for (int i = 0; i < EJ_N; i++) y[i] = ok ? y[i] * r : 0.0;
            if (step >= 0) {
#pragma unroll
                for (int i = 0; i < EJ_N; i++) sm.q[i] = y[i];
            }
        }
        if (step < 0) continue;
        __syncwarp();
        double q[EJ_N];
        load25(sm.q, q);
        const double s = lane > g ? fma(q[0], y[0], dot24(q, y)) : 0.0;
#pragma unroll
        for (int i = 0; i < EJ_N; i++) y[i] = fma(-s, q[i], y[i]);
        __syncwarp();
    }
    // ---- 6. select_pca_basis. When every eigenvalue is kept (the usual
    //         case) it reduces to signing each column by its largest-magnitude
    //         entry (first on ties), with the same result
    const double lam0 = sm.lam[0] > 0.0 ? sm.lam[0] : 0.0;
    bool all_kept = lam0 > 0.0;
#pragma unroll
    for (int k = 0; k < EJ_TOP; k++) all_kept = all_kept && sm.lam[k] > 1e-9 * lam0;
    if (all_kept) {
        double mx = fabs(y[0]);
        bool neg = y[0] < 0.0;
#pragma unroll
        for (int r = 1; r < EJ_N; r++)
            if (fabs(y[r]) > mx) {
                mx = fabs(y[r]);
                neg = y[r] < 0.0;
            }
        if (lane < EJ_TOP) {
#pragma unroll
            for (int r = 0; r < EJ_N; r++) basis[r * EJ_TOP + lane] = float(neg ? -y[r] : y[r]);
        }
    } else {
        if (lane < EJ_TOP) {
#pragma unroll
            for (int r = 0; r < EJ_N; r++) sm.Z[r][lane] = y[r];
        }
        __syncwarp();
        if (lane == 0) {
            double ev[EJ_TOP];
            for (int k = 0; k < EJ_TOP; k++) ev[k] = sm.lam[k];
            select_pca_basis(ev, &sm.Z[0][0], EJ_TOP + 1, sm.work, basis);
        }
    }
    __syncwarp();
    if (lane == 0 && status) *status = sm.bad ? -1 : EJ_INV_ITERS;
}


}  // namespace gls
