// gls_surf.cu — registration and fusion on the GPU: RawChannels, the SURF
// integral image, fast-Hessian detector, orientation + 64-D descriptor,
// brute-force matching, RANSAC + least-squares homography, and the
// registerAndFuse / registerImage warps, behind the gls_surf_* / gls_*
// entry points of include/glscam.h.
//
// Reference: ImageRegistration/SURF.metal, SURF.cpp, Homography.cpp,
// LeastSquaresHomography.cpp, RTL/RANSAC.hpp, PyramidFusion/pyramidFusion.cpp.
// Every float expression that decides a keypoint, a descriptor or a model
// is evaluated with one IEEE rounding per operation (gls_fmath.h), so the
// results are bit-identical to the CPU restatement that checks them.
//
// Layout in HBM per detector: the integral image (W+1) x (H+1) F32 and its
// transposed column sums (W x H); 64000 candidate keypoints; per feature
// slot the kept keypoints (28 B) and descriptors (256 B). The detector
// computes Hessian determinants tile by tile in shared memory and runs the
// 3x3x3 non-maximum suppression on them in the same kernel, so no
// determinant plane is ever written to HBM.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <random>
#include <set>
#include <type_traits>
#include <vector>

#include "gls_common.cuh"
#include "gls_devbuf.h"
#include "gls_fmath.h"
#include "gls_kernels.h"
#include "gls_warp.cuh"

namespace gls {

using glsm::dadd;
using glsm::ddiv;
using glsm::dmul;
using glsm::dsqrt;
using glsm::dsub;
using glsm::fadd;
using glsm::fdiv;
using glsm::fmul;
using glsm::fsqrt;
using glsm::fsub;
using glsm::gls_atan2f;
using glsm::gls_cosf;
using glsm::gls_sinf;

constexpr int kMaxKeypoints = GLS_SURF_MAX_KEYPOINTS;
constexpr int kMaxOctaves = 6;
constexpr int kLayers = 4;  // nOctaveLayers + 2 with nOctaveLayers = 2 (the only layer count served)

// ------------------------------------------------------------ host: patterns
struct Box {
    int x1, y1, x2, y2;
    float w;
};

// resizeHaarPattern (SURF.cpp:103-114)
template <int N>
static void resize_haar(const int src[][5], Box* dst, int old_size, int new_size) {
    const float ratio = float(new_size) / float(old_size);
    for (int k = 0; k < N; k++) {
        const int dx1 = int(std::lrint(ratio * float(src[k][0])));
        const int dy1 = int(std::lrint(ratio * float(src[k][1])));
        const int dx2 = int(std::lrint(ratio * float(src[k][2])));
        const int dy2 = int(std::lrint(ratio * float(src[k][3])));
        dst[k] = {dx1, dy1, dx2, dy2, float(src[k][4]) / (float(dx2 - dx1) * float(dy2 - dy1))};
    }
}

// One Hessian layer: the box corners the Metal kernel reads (gpuSurfHF,
// SURF.cpp:200-225) and its margin crop (DetAndTraceHaarPattern,
// SURF.cpp:235-265).
struct LayerDev {
    short dx[8][2];   // r02 r07 r32 r37 | r62 r67 r92 r97 (x, y)
    short dy[8][2];   // r20 r23 r70 r73 | r26 r76 r29 r79
    short dxy[4][4][2];
    float w, wxy;
    int mx, my, mw, mh;
    int size;
};

struct OctaveDev {
    LayerDev layer[kLayers];
    int step, lw, lh;      // layer grid = image / step
    int tiles_x, tiles_y;  // detector tiles over the layer grid
    int block0;            // first block of this octave
};

struct DetectArgs {
    OctaveDev oct[kMaxOctaves];
    int n_oct;
    const float* sum;
    int sum_pitch;  // floats
    int sum_w, sum_h;
    float threshold;
    int per_axis;  // corrected interpolation (else the reference's scale-offset broadcast)
    gls_keypoint* cand;
    int* cand_count;
};

static LayerDev make_layer(int sum_w, int sum_h, int size, int step) {
    static const int dx_s[3][5] = {{0, 2, 3, 7, 1}, {3, 2, 6, 7, -2}, {6, 2, 9, 7, 1}};
    static const int dy_s[3][5] = {{2, 0, 7, 3, 1}, {2, 3, 7, 6, -2}, {2, 6, 7, 9, 1}};
    static const int dxy_s[4][5] = {{1, 1, 4, 4, 1}, {5, 1, 8, 4, -1}, {1, 5, 4, 8, -1}, {5, 5, 8, 8, 1}};
    Box bx[3], by[3], bxy[4];
    resize_haar<3>(dx_s, bx, 9, size);
    resize_haar<3>(dy_s, by, 9, size);
    resize_haar<4>(dxy_s, bxy, 9, size);
    LayerDev L{};
    auto set = [](short* d, int x, int y) {
        d[0] = short(x);
        d[1] = short(y);
    };
    set(L.dx[0], bx[0].x1, bx[0].y1);
    set(L.dx[1], bx[0].x1, bx[0].y2);
    set(L.dx[2], bx[0].x2, bx[0].y1);
    set(L.dx[3], bx[0].x2, bx[0].y2);
    set(L.dx[4], bx[1].x2, bx[1].y1);
    set(L.dx[5], bx[1].x2, bx[1].y2);
    set(L.dx[6], bx[2].x2, bx[2].y1);
    set(L.dx[7], bx[2].x2, bx[2].y2);
    set(L.dy[0], by[0].x1, by[0].y1);
    set(L.dy[1], by[0].x1, by[0].y2);
    set(L.dy[2], by[0].x2, by[0].y1);
    set(L.dy[3], by[0].x2, by[0].y2);
    set(L.dy[4], by[1].x1, by[1].y2);
    set(L.dy[5], by[1].x2, by[1].y2);
    set(L.dy[6], by[2].x1, by[2].y2);
    set(L.dy[7], by[2].x2, by[2].y2);
    for (int k = 0; k < 4; k++) {
        set(L.dxy[k][0], bxy[k].x1, bxy[k].y1);
        set(L.dxy[k][1], bxy[k].x1, bxy[k].y2);
        set(L.dxy[k][2], bxy[k].x2, bxy[k].y1);
        set(L.dxy[k][3], bxy[k].x2, bxy[k].y2);
    }
    L.w = bx[0].w;
    L.wxy = bxy[0].w;
    L.mx = (size / 2) / step;
    L.my = (size / 2) / step;
    L.mw = 1 + (sum_w - 1 - size) / step;
    L.mh = 1 + (sum_h - 1 - size) / step;
    if (size > sum_w - 1 || size > sum_h - 1) L.mw = L.mh = 0;  // the wavelet does not fit: no samples
    L.size = size;
    return L;
}

// ------------------------------------------------------------ device: Hessian
__device__ __forceinline__ float rect_gpu(float tr, float tl, float br, float bl) {
    return fsub(fadd(0.5f, fsub(tr, tl)), fsub(br, bl));
}

// calcHaarPatternDx / Dy / Dxy + calcDetAndTrace (SURF.metal:77-145)
__device__ __forceinline__ void det_trace_at(const float* __restrict__ S, int pitch, int px, int py,
                                             const LayerDev& L, float* det, float* trace) {
    auto rd = [&](const short* o) { return __ldg(S + size_t(py + o[1]) * pitch + px + o[0]); };
    const float r02 = rd(L.dx[0]), r07 = rd(L.dx[1]), r32 = rd(L.dx[2]), r37 = rd(L.dx[3]);
    const float r62 = rd(L.dx[4]), r67 = rd(L.dx[5]), r92 = rd(L.dx[6]), r97 = rd(L.dx[7]);
    const float dx = fmul(L.w, fsub(rect_gpu(r97, r92, r07, r02), fmul(3.0f, rect_gpu(r67, r62, r37, r32))));
    const float r20 = rd(L.dy[0]), r23 = rd(L.dy[1]), r70 = rd(L.dy[2]), r73 = rd(L.dy[3]);
    const float r26 = rd(L.dy[4]), r76 = rd(L.dy[5]), r29 = rd(L.dy[6]), r79 = rd(L.dy[7]);
    const float dy = fmul(L.w, fsub(rect_gpu(r79, r70, r29, r20), fmul(3.0f, rect_gpu(r76, r73, r26, r23))));
    float dxy = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float wk = (k == 0 || k == 3) ? L.wxy : -L.wxy;
        const float p0 = rd(L.dxy[k][0]), p1 = rd(L.dxy[k][1]), p2 = rd(L.dxy[k][2]), p3 = rd(L.dxy[k][3]);
        dxy = fadd(dxy, fmul(wk, rect_gpu(p0, p1, p2, p3)));
    }
    *det = fsub(fmul(dx, dy), fmul(fmul(0.81f, dxy), dxy));
    *trace = fadd(dx, dy);
}

__device__ __forceinline__ float det3(const float a[3], const float b[3], const float c[3]) {
    const float cx = fsub(fmul(b[1], c[2]), fmul(b[2], c[1]));
    const float cy = fsub(fmul(b[2], c[0]), fmul(b[0], c[2]));
    const float cz = fsub(fmul(b[0], c[1]), fmul(b[1], c[0]));
    return fadd(fadd(fmul(a[0], cx), fmul(a[1], cy)), fmul(a[2], cz));
}

// A detector tile: 64 x 32 samples, NMS positions the 62 x 30 inside. A thread
// evaluates 8 rows of a column, so that a box corner's address is formed once
// for 8 samples; the first octave's tiles (three quarters of all samples) read
// the corners from the integral image's region in shared memory, one wavefront
// a read where the unaligned global read takes two, the later octaves' regions
// do not fit.
constexpr int DS_X = 64, DS_Y = 32, DS_R = 8;
constexpr int DT_X = DS_X - 2, DT_Y = DS_Y - 2;
constexpr int DR_W = DS_X + 27, DR_H = DS_Y + 27;  // region of the first octave: its largest wavelet spans 27

struct DetectSmem {
    int4 corner[kLayers][8];  // corner offsets of the 8 boxes, in rect_gpu's order
    float det[kLayers][DS_Y][DS_X];
    float sum[DR_H][DR_W];
};

// calcHaarPatternDx / Dy / Dxy + the determinant (SURF.metal:77-145) of DS_R
// samples, `dy` floats apart.
__device__ __forceinline__ void det_column(const float* __restrict__ p, const int4 (&corner)[8], int dy, float w,
                                           float wxy, float (&det)[DS_R]) {
    auto box = [&](int k, float (&v)[DS_R]) {
        const int4 c = corner[k];
        const float *q0 = p + c.x, *q1 = p + c.y, *q2 = p + c.z, *q3 = p + c.w;
#pragma unroll
        for (int r = 0; r < DS_R; r++) v[r] = rect_gpu(q0[r * dy], q1[r * dy], q2[r * dy], q3[r * dy]);
    };
    float u[DS_R], v[DS_R], dx[DS_R];
    box(0, u);
    box(1, v);
#pragma unroll
    for (int r = 0; r < DS_R; r++) dx[r] = fmul(w, fsub(u[r], fmul(3.0f, v[r])));
    box(2, u);
    box(3, v);
#pragma unroll
    for (int r = 0; r < DS_R; r++) det[r] = fmul(dx[r], fmul(w, fsub(u[r], fmul(3.0f, v[r]))));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        box(4 + k, u);
#pragma unroll
        for (int r = 0; r < DS_R; r++)
            v[r] = fadd(k == 0 ? 0.0f : v[r], fmul(k == 0 || k == 3 ? wxy : -wxy, u[r]));
    }
#pragma unroll
    for (int r = 0; r < DS_R; r++) det[r] = fsub(det[r], fmul(fmul(0.81f, v[r]), v[r]));
}

// A feature slot's count, set from a host value (gls_surf_load_features).
__global__ void k_store_count(int* count, int n) { *count = n; }

// calcDetAndTrace for the four layers of an octave over a tile plus a
// one-sample halo, into shared memory; then findMaximaInLayer
// (SURF.metal:249-313) with interpolateKeypoint (:207-247) for the two
// middle layers. Determinants outside a layer's margin crop are 0, as an
// unwritten determinant plane.
//
// What bounds it: 32 corner reads and some 90 instructions a sample and layer.
// 2016x1512: 171 us; 423 when every sample formed its corners' addresses (480
// instructions a sample, tiles of 32 x 8 positions).
__global__ void __launch_bounds__(256) k_hessian_nms(DetectArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DetectSmem& sm = *reinterpret_cast<DetectSmem*>(smem_raw);
    auto& det = sm.det;
    // the later octaves first: their blocks take the longest
    const int block = gridDim.x - 1 - blockIdx.x;
    int o = 0;
    while (o + 1 < a.n_oct && block >= a.oct[o + 1].block0) o++;
    const OctaveDev& O = a.oct[o];
    const int b = block - O.block0;
    const int bx = b % O.tiles_x, by = b / O.tiles_x;
    const int x0 = bx * DT_X - 1, y0 = by * DT_Y - 1;  // first sample
    const int step = O.step;
    const int tx = threadIdx.x % DS_X, ty = threadIdx.x / DS_X * DS_R;
    // first octave: layer l reads [x - (4 + 3 l), x + 5 + 3 l], at most 13 before and 14 after
    const int rx = x0 - 13, ry = y0 - 13;
    if (o == 0) {
        for (int i = threadIdx.x; i < DR_W * DR_H; i += 256) {
            const int x = rx + i % DR_W, y = ry + i / DR_W;
            (&sm.sum[0][0])[i] = x >= 0 && x < a.sum_w && y >= 0 && y < a.sum_h ? __ldg(a.sum + size_t(y) * a.sum_pitch + x) : 0.0f;
        }
    }
    if (threadIdx.x < kLayers * 32) {
        const int l = threadIdx.x / 32, e = threadIdx.x % 32;
        const LayerDev& L = O.layer[l];
        // r97 r92 r07 r02, r67 r62 r37 r32; r79 r70 r29 r20, r76 r73 r26 r23
        const int order = int((0x1435062723450167ull >> (4 * (e % 16))) & 15);
        const short* c = e < 8 ? L.dx[order] : e < 16 ? L.dy[order] : L.dxy[(e - 16) / 4][e % 4];
        reinterpret_cast<int*>(sm.corner[l])[e] = c[1] * (o == 0 ? DR_W : a.sum_pitch) + c[0];
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < kLayers; l++) {
        const LayerDev& L = O.layer[l];
        const int ix = x0 + tx - L.mx, iy = y0 + ty - L.my;
        float d[DS_R];
        const bool col = ix >= 0 && ix < L.mw;
        if (o == 0) {
            det_column(&sm.sum[y0 + ty - L.my - ry][x0 + tx - L.mx - rx], sm.corner[l], DR_W, L.w, L.wxy, d);
        } else if (col && iy >= 0 && iy + DS_R <= L.mh) {
            det_column(a.sum + size_t(iy * step) * a.sum_pitch + ix * step, sm.corner[l], step * a.sum_pitch, L.w, L.wxy,
                       d);
        } else {
#pragma unroll 1
            for (int r = 0; r < DS_R; r++) {
                float v = 0.0f, t;
                if (col && iy + r >= 0 && iy + r < L.mh)
                    det_trace_at(a.sum, a.sum_pitch, ix * step, (iy + r) * step, L, &v, &t);
                det[l][ty + r][tx] = v;
            }
            continue;
        }
#pragma unroll
        for (int r = 0; r < DS_R; r++) det[l][ty + r][tx] = col && iy + r >= 0 && iy + r < L.mh ? d[r] : 0.0f;
    }
    __syncthreads();
    const int x = x0 + tx;
    if (tx < 1 || tx > DT_X) return;
#pragma unroll 1
    for (int k = 0; k < 2 * DS_R; k++) {
        const int l = 1 + k % 2, sy = ty + k / 2, y = y0 + sy;
        if (sy < 1 || sy > DT_Y) continue;
        const float v = det[l][sy][tx];
        if (!(v > a.threshold)) continue;
        const LayerDev& L = O.layer[l];
        const int margin = (O.layer[l + 1].size / 2) / step + 1;
        if (x < margin || x >= O.lw - margin || y < margin || y >= O.lh - margin) continue;
        bool mx = true;
        for (int i = 0; i < 3 && mx; i++)
            for (int dy = -1; dy <= 1 && mx; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    if (i == 1 && dx == 0 && dy == 0) continue;
                    if (!(v > det[l - 1 + i][sy + dy][tx + dx])) {
                        mx = false;
                        break;
                    }
                }
        if (!mx) continue;
        auto n9 = [&](int i, int dy, int dx) { return det[l - 1 + i][sy + dy][tx + dx]; };
        const int size = L.size, s0 = O.layer[l - 1].size;
        const int sum_y = step * (y - (size / 2) / step);
        const int sum_x = step * (x - (size / 2) / step);
        float dtmp, tr = 0.0f;  // trace plane value; 0 outside the crop, as unwritten
        if (x - L.mx < L.mw && y - L.my < L.mh)
            det_trace_at(a.sum, a.sum_pitch, (x - L.mx) * step, (y - L.my) * step, L, &dtmp, &tr);
        gls_keypoint kp;
        kp.x = fadd(float(sum_x), fmul(float(size - 1), 0.5f));
        kp.y = fadd(float(sum_y), fmul(float(size - 1), 0.5f));
        kp.size = float(size);
        kp.angle = -1.0f;
        kp.response = v;
        kp.octave = o;
        kp.class_id = tr > 0.0f ? 1 : 0;
        const float B[3] = {-fdiv(fsub(n9(1, 0, 1), n9(1, 0, -1)), 2.0f), -fdiv(fsub(n9(1, 1, 0), n9(1, -1, 0)), 2.0f),
                            -fdiv(fsub(n9(2, 0, 0), n9(0, 0, 0)), 2.0f)};
        const float dxx = fadd(fsub(n9(1, 0, -1), fmul(2.0f, n9(1, 0, 0))), n9(1, 0, 1));
        const float dxy = fdiv(fadd(fsub(fsub(n9(1, 1, 1), n9(1, 1, -1)), n9(1, -1, 1)), n9(1, -1, -1)), 4.0f);
        const float dxs = fdiv(fadd(fsub(fsub(n9(2, 0, 1), n9(2, 0, -1)), n9(0, 0, 1)), n9(0, 0, -1)), 4.0f);
        const float dyy = fadd(fsub(n9(1, -1, 0), fmul(2.0f, n9(1, 0, 0))), n9(1, 1, 0));
        const float dys = fdiv(fadd(fsub(fsub(n9(2, 1, 0), n9(2, -1, 0)), n9(0, 1, 0)), n9(0, -1, 0)), 4.0f);
        const float dss = fadd(fsub(n9(0, 0, 0), fmul(2.0f, n9(1, 0, 0))), n9(2, 0, 0));
        const float A0[3] = {dxx, dxy, dxs}, A1[3] = {dxy, dyy, dys}, A2[3] = {dxs, dys, dss};
        float X[3] = {0.0f, 0.0f, 0.0f};
        const float dt = det3(A0, A1, A2);
        if (dt != 0.0f) {  // solve3x3 (SURF.metal:189-205)
            X[2] = fdiv(det3(A0, A1, B), dt);
            if (a.per_axis) {
                X[0] = fdiv(det3(B, A1, A2), dt);
                X[1] = fdiv(det3(A0, B, A2), dt);
            } else {  // `(float3)(a, b, c) / det` is float3(c) / det: the scale offset in every lane
                X[0] = X[1] = X[2];
            }
        }
        const bool all_zero = X[0] == 0.0f && X[1] == 0.0f && X[2] == 0.0f;
        if (all_zero || !(fabsf(X[0]) <= 1.0f && fabsf(X[1]) <= 1.0f && fabsf(X[2]) <= 1.0f)) continue;
        kp.x = fadd(kp.x, fmul(X[0], float(step)));
        kp.y = fadd(kp.y, fmul(X[1], float(step)));
        kp.size = rintf(fadd(kp.size, fmul(X[2], float(size - s0))));
        const int idx = atomicAdd(a.cand_count, 1);
        if (idx < kMaxKeypoints) a.cand[idx] = kp;
    }
}

// KeypointGreater (SURF.cpp:1215-1227), with the candidate index as the
// last key so that the order is total.
__device__ __forceinline__ bool kp_before(const gls_keypoint& a, int ia, const gls_keypoint& b, int ib) {
    if (a.response != b.response) return a.response > b.response;
    if (a.size != b.size) return a.size > b.size;
    if (a.octave != b.octave) return a.octave > b.octave;
    if (a.y != b.y) return a.y > b.y;
    if (a.x != b.x) return a.x < b.x;
    return ia < ib;
}

// Rank sort of the candidates and the max_features cut (SURF.cpp:1285,
// 1413-1418): candidate i goes to its rank if the rank is below keep. Bound by
// its n^2 comparisons: a block ranks 16 candidates, 16 threads each over every
// 16th four others, on the responses alone; a candidate whose response is not
// its own alone compares the further keys in a second sweep. 7000 candidates:
// 21 us, 278 with a thread a candidate (28 blocks) and the full comparison.
constexpr int kRankPer = 16, kRankLanes = 16;
__global__ void __launch_bounds__(kRankPer * kRankLanes)
    k_keypoint_rank(const gls_keypoint* __restrict__ cand, const int* __restrict__ cand_count, int keep,
                    gls_keypoint* __restrict__ out, int* __restrict__ out_count) {
    constexpr int N = 4 * kRankPer * kRankLanes;
    __shared__ float4 tile[N / 4];
    const int n = min(*cand_count, kMaxKeypoints);
    if (blockIdx.x == 0 && threadIdx.x == 0) *out_count = min(n, keep);
    if (blockIdx.x * kRankPer >= n) return;  // whole block past the end (block-uniform)
    const int i = blockIdx.x * kRankPer + threadIdx.x / kRankLanes, lane = threadIdx.x % kRankLanes;
    gls_keypoint me{};
    if (i < n) me = cand[i];
    const float key = me.response;
    int rank = 0, equal = 0;
    for (int j0 = 0; j0 < n; j0 += N) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {  // past the end: behind every candidate
            const int j = threadIdx.x + k * (N / 4);
            reinterpret_cast<float*>(tile)[j] = j0 + j < n ? cand[j0 + j].response : -INFINITY;
        }
        __syncthreads();
#pragma unroll 8
        for (int j = lane; j < N / 4; j += kRankLanes) {
            const float4 r = tile[j];
            rank += (r.x > key) + (r.y > key) + (r.z > key) + (r.w > key);
            equal += (r.x == key) + (r.y == key) + (r.z == key) + (r.w == key);
        }
    }
#pragma unroll
    for (int o = kRankLanes / 2; o > 0; o >>= 1) equal += __shfl_xor_sync(0xffffffffu, equal, o);
    if (i < n && equal > 1)  // not only itself: the further keys decide
        for (int j = lane; j < n; j += kRankLanes) {
            const gls_keypoint c = cand[j];
            if (c.response == key && kp_before(c, j, me, i)) rank++;
        }
#pragma unroll
    for (int o = kRankLanes / 2; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (lane == 0 && i < n && rank < keep) out[rank] = me;
}

// ------------------------------------------------------------ descriptors
struct DescTables {  // SURFInvoker constructor (SURF.cpp:466-497)
    float apt_x[169], apt_y[169], aptw[169];
    float dw[400];
    int n_ori;
};

__device__ __forceinline__ float rect_cpu(float tr, float tl, float br, float bl) {
    // SURF.cpp:79-82: the 0.5 is a double literal
    return __double2float_rn(dsub(dadd(0.5, double(fsub(tr, tl))), double(fsub(br, bl))));
}

// calcHaarPattern (SURF.cpp:84-101) over two boxes
__device__ __forceinline__ float haar2(const float* __restrict__ S, int pitch, int px, int py, const Box* f) {
    float d = 0.0f;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const Box& b = f[k];
        const float p0 = __ldg(S + size_t(py + b.y1) * pitch + px + b.x1);
        const float p1 = __ldg(S + size_t(py + b.y2) * pitch + px + b.x1);
        const float p2 = __ldg(S + size_t(py + b.y1) * pitch + px + b.x2);
        const float p3 = __ldg(S + size_t(py + b.y2) * pitch + px + b.x2);
        d = fadd(d, fmul(b.w, rect_cpu(p0, p1, p2, p3)));
    }
    return d;
}

__device__ void resize_haar2_dev(const int (*src)[5], Box* dst, int new_size) {
    const float ratio = fdiv(float(new_size), 4.0f);
    for (int k = 0; k < 2; k++) {
        const int dx1 = lrintf(fmul(ratio, float(src[k][0])));
        const int dy1 = lrintf(fmul(ratio, float(src[k][1])));
        const int dx2 = lrintf(fmul(ratio, float(src[k][2])));
        const int dy2 = lrintf(fmul(ratio, float(src[k][3])));
        dst[k] = {dx1, dy1, dx2, dy2, fdiv(float(src[k][4]), fmul(float(dx2 - dx1), float(dy2 - dy1)))};
    }
}

struct DescArgs {
    const float* img;
    int img_pitch, iw, ih;
    const float* sum;
    int sum_pitch, sw, sh;
    const DescTables* tab;
    gls_keypoint* kps;
    const int* count;
    float* desc;
    int all;  // describe every keypoint (else the reference's ranges, SURF.cpp:681-693)
};

constexpr int kDescThreads = 128;
constexpr int kMaxWinIdx = 42;  // rows / columns of the window resizeVV reads

// SURFInvoker::computeRange for one keypoint per block (SURF.cpp:499-677):
// dominant orientation over the Haar responses in a radius-6s disc, the
// rotated window (only the 42 x 42 of its pixels that resizeVV reads,
// each at the position the reference's running sums reach), the 21 x 21
// patch, 20 x 20 gradients and the 4 x 4 x 4 descriptor.
// Bound by the latency of its serial parts: all blocks of 1500 keypoints run at
// once, and the largest wavelet's window has 600 rows and columns of running
// sums. Those loops add only; the pixels are gathered afterwards by all threads.
// 1500 keypoints of a 2016x1512 image: 58 us (125 with the gather inside the
// column loops and serial scans of the samples and bins).
__global__ void __launch_bounds__(kDescThreads) k_describe(DescArgs a) {
    const int k = blockIdx.x;
    const int n = *a.count;
    if (k >= n) return;
    // SURFInvoker::run cuts K > 32 keypoints into ceil(K/8) ranges of
    // ceil(K/8): the first min(K, ceil(K/8)^2) are described, the others keep
    // angle -1 and a zero descriptor
    const int r8 = (n + 7) / 8;
    if (!a.all && n > 32 && k >= r8 * r8) {
        for (int i = threadIdx.x; i < 64; i += blockDim.x) a.desc[size_t(k) * 64 + i] = 0.0f;
        return;
    }
    __shared__ float X[169], Y[169], ANG[169];
    __shared__ float bx_s[72], by_s[72], mod_s[72];
    __shared__ float rowx[kMaxWinIdx], rowy[kMaxWinIdx];
    __shared__ int q[kMaxWinIdx];
    __shared__ float M[kMaxWinIdx][kMaxWinIdx + 1], PY[kMaxWinIdx][kMaxWinIdx + 1];
    __shared__ int n_valid[2][kDescThreads / 32];
    __shared__ float P[21][22];
    __shared__ float DX[20][21], DY[20][21];
    __shared__ float cell[16][4];
    __shared__ Box dxt[2], dyt[2];
    __shared__ float dir_s;
    const DescTables& T = *a.tab;
    const int t = threadIdx.x;
    gls_keypoint kp = a.kps[k];
    float* desc = a.desc + size_t(k) * 64;
    for (int i = t; i < 64; i += blockDim.x) desc[i] = 0.0f;
    const float s = fdiv(fmul(kp.size, 1.2f), 9.0f);
    const int gws = 2 * lrintf(fmul(2.0f, s));
    if (a.sh < gws || a.sw < gws) {
        if (t == 0) a.kps[k].size = -1.0f;
        return;
    }
    if (t == 0) {
        const int dx_s[2][5] = {{0, 0, 2, 4, -1}, {2, 0, 4, 4, 1}};
        const int dy_s[2][5] = {{0, 0, 4, 2, 1}, {0, 2, 4, 4, -1}};
        resize_haar2_dev(dx_s, dxt, gws);
        resize_haar2_dev(dy_s, dyt, gws);
    }
    __syncthreads();
    // orientation samples, compacted in the reference's sample order
    const float half_wav = fdiv(float(gws - 1), 2.0f);
    int valid[2] = {0, 0};
    float vxs[2], vys[2];
    for (int r = 0; r < 2; r++) {
        const int kk = t + r * kDescThreads;
        if (kk >= T.n_ori) continue;
        const int x = lrintf(fsub(fadd(kp.x, fmul(T.apt_x[kk], s)), half_wav));
        const int y = lrintf(fsub(fadd(kp.y, fmul(T.apt_y[kk], s)), half_wav));
        if (y < 0 || y >= a.sh - gws || x < 0 || x >= a.sw - gws) continue;
        vxs[r] = haar2(a.sum, a.sum_pitch, x, y, dxt);
        vys[r] = haar2(a.sum, a.sum_pitch, x, y, dyt);
        valid[r] = 1;
    }
    unsigned ballot[2];
    for (int r = 0; r < 2; r++) {
        ballot[r] = __ballot_sync(0xffffffffu, valid[r]);
        if (t % 32 == 0) n_valid[r][t / 32] = __popc(ballot[r]);
    }
    __syncthreads();
    int nangle = 0;
    for (int r = 0; r < 2; r++) {
        int j = nangle;  // samples before this thread's
        for (int w = 0; w < kDescThreads / 32; w++) {
            if (w < t / 32) j += n_valid[r][w];
            nangle += n_valid[r][w];
        }
        j += __popc(ballot[r] & ((1u << (t % 32)) - 1));
        const int kk = t + r * kDescThreads;
        if (!valid[r]) continue;
        const float xv = fmul(vxs[r], T.aptw[kk]), yv = fmul(vys[r], T.aptw[kk]);
        X[j] = xv;
        Y[j] = yv;
        const float tdeg = __double2float_rn(dmul(double(gls_atan2f(yv, xv)), 180.0 / 3.14159265358979323846));
        ANG[j] = float(lrintf(tdeg < 0.0f ? fadd(tdeg, 360.0f) : tdeg));
    }
    __syncthreads();
    if (nangle == 0) {
        if (t == 0) a.kps[k].size = -1.0f;
        return;
    }
    if (t < 72) {
        const float bin = float(5 * t);
        float sx = 0.0f, sy = 0.0f;
        for (int j = 0; j < nangle; j++) {
            const float d = fabsf(fsub(ANG[j], bin));
            if (d < 30.0f || d > 330.0f) {
                sx = fadd(sx, X[j]);
                sy = fadd(sy, Y[j]);
            }
        }
        bx_s[t] = sx;
        by_s[t] = sy;
        mod_s[t] = fadd(fmul(sx, sx), fmul(sy, sy));
    }
    __syncthreads();
    if (t < 32) {  // the first bin with the largest modulus above 0
        float best = 0.0f;
        int bin = 72;
        for (int b = t; b < 72; b += 32)
            if (mod_s[b] > best) {
                best = mod_s[b];
                bin = b;
            }
        for (int o = 16; o > 0; o >>= 1) {
            const float m = __shfl_xor_sync(0xffffffffu, best, o);
            const int b = __shfl_xor_sync(0xffffffffu, bin, o);
            if (m > best || (m == best && b < bin)) {
                best = m;
                bin = b;
            }
        }
        if (t == 0) {
            dir_s = bin < 72 ? gls_atan2f(-by_s[bin], bx_s[bin]) : gls_atan2f(-0.0f, 0.0f);
            a.kps[k].angle = dir_s;
        }
    }
    __syncthreads();
    const float dir = fmul(dir_s, float(3.14159265358979323846 / 180.0));
    const float sin_dir = -gls_sinf(dir);
    const float cos_dir = gls_cosf(dir);
    const int win = int(fmul(21.0f, s));
    const float dsize = fdiv(float(win), 21.0f);
    if (t < 21) {
        const int qi = int(fmul(float(t), dsize));
        q[2 * t] = qi;
        q[2 * t + 1] = qi + 1;
    }
    __syncthreads();
    if (t == 0) {  // row starts: the running sums of the window's outer loop
        const float off = -fdiv(float(win - 1), 2.0f);
        float sx = fadd(fadd(kp.x, fmul(off, cos_dir)), fmul(off, sin_dir));
        float sy = fadd(fsub(kp.y, fmul(off, sin_dir)), fmul(off, cos_dir));
        int r = 0;  // the indices do not decrease: dsize > 1 for every keypoint
        for (int need = 0; need < kMaxWinIdx; need++) {
#pragma unroll 4
            for (const int end = q[need]; r < end; r++) {
                sx = fadd(sx, sin_dir);
                sy = fadd(sy, cos_dir);
            }
            rowx[need] = sx;
            rowy[need] = sy;
        }
    }
    __syncthreads();
    if (t < kMaxWinIdx) {  // one requested window row per thread
        float px = rowx[t], py = rowy[t];
        int c = 0;
        for (int need = 0; need < kMaxWinIdx; need++) {
#pragma unroll 4
            for (const int end = q[need]; c < end; c++) {
                px = fadd(px, cos_dir);
                py = fsub(py, sin_dir);
            }
            M[t][need] = px;
            PY[t][need] = py;
        }
    }
    __syncthreads();
    for (int e = t; e < kMaxWinIdx * kMaxWinIdx; e += blockDim.x) {
        const int ncols1 = a.iw - 1, nrows1 = a.ih - 1;
        const float px = M[e / kMaxWinIdx][e % kMaxWinIdx], py = PY[e / kMaxWinIdx][e % kMaxWinIdx];
        const int ix = int(floorf(px)), iy = int(floorf(py));
        float v;
        if (unsigned(ix) < unsigned(ncols1) && unsigned(iy) < unsigned(nrows1)) {
            const float fa = fsub(px, float(ix)), fb = fsub(py, float(iy));
            const float oa = fsub(1.0f, fa), ob = fsub(1.0f, fb);
            const float* r0 = a.img + size_t(iy) * a.img_pitch;
            const float* r1 = r0 + a.img_pitch;
            const float top = fadd(fmul(__ldg(r0 + ix), oa), fmul(__ldg(r0 + ix + 1), fa));
            const float bot = fadd(fmul(__ldg(r1 + ix), oa), fmul(__ldg(r1 + ix + 1), fa));
            v = roundf(fadd(fmul(top, ob), fmul(bot, fb)));
        } else {
            const int xx = min(max(int(roundf(px)), 0), ncols1);
            const int yy = min(max(int(roundf(py)), 0), nrows1);
            v = __ldg(a.img + size_t(yy) * a.img_pitch + xx);
        }
        M[e / kMaxWinIdx][e % kMaxWinIdx] = v;
    }
    __syncthreads();
    for (int e = t; e < 441; e += blockDim.x) {  // resizeVV (SURF.cpp:427-446)
        const int i = e / 21, j = e % 21;
        const float fi = fmul(float(i), dsize), fj = fmul(float(j), dsize);
        const int ii = int(fi), jj = int(fj);
        const float id = fsub(fi, float(ii)), jd = fsub(fj, float(jj));
        float v = 0.0f;
        if (jj < win - 1 && ii < win - 1) {
            const float oi = fsub(1.0f, id), oj = fsub(1.0f, jd);
            v = fmul(fmul(oi, oj), M[2 * i][2 * j]);
            v = fadd(v, fmul(fmul(id, oj), M[2 * i + 1][2 * j]));
            v = fadd(v, fmul(fmul(jd, oi), M[2 * j][2 * j + 1]));
            v = fadd(v, fmul(fmul(id, jd), M[2 * i + 1][2 * j + 1]));
        }
        P[i][j] = v;
    }
    __syncthreads();
    for (int e = t; e < 400; e += blockDim.x) {
        const int i = e / 20, j = e % 20;
        const float dw = T.dw[e];
        DX[i][j] = fmul(fsub(fadd(fsub(P[i][j + 1], P[i][j]), P[i + 1][j + 1]), P[i + 1][j]), dw);
        DY[i][j] = fmul(fsub(fadd(fsub(P[i + 1][j], P[i][j]), P[i + 1][j + 1]), P[i][j + 1]), dw);
    }
    __syncthreads();
    if (t < 64) {  // sums of dx, dy, |dx|, |dy| of a cell, one each
        const int ci = t / 16, cj = t / 4 % 4, m = t % 4;
        float sum = 0.0f;
        for (int y = ci * 5; y < ci * 5 + 5; y++)
#pragma unroll
            for (int x = cj * 5; x < cj * 5 + 5; x++) {
                const float v = m & 1 ? DY[y][x] : DX[y][x];
                sum = fadd(sum, m & 2 ? fabsf(v) : v);
            }
        cell[t / 4][m] = sum;
    }
    __syncthreads();
    __shared__ float scale_s;
    if (t == 0) {
        float sq = 0.0f;
        for (int c = 0; c < 16; c++)
            for (int m = 0; m < 4; m++) sq = fadd(sq, fmul(cell[c][m], cell[c][m]));
        scale_s = __double2float_rn(ddiv(1.0, double(fadd(fsqrt(sq), FLT_EPSILON))));
    }
    __syncthreads();
    if (t < 64) desc[t] = fmul(cell[t / 4][t % 4], scale_s);
}

// ------------------------------------------------------------ matching
// A batch of matching / homography jobs: each pairs a query slot (the
// reference frame's features) with a train slot; blockIdx.y is the job.
constexpr int kMaxJobs = 64;
struct MatchJob {
    const float* d1;
    const int* n1;
    const gls_keypoint* k1;
    const float* d2;
    const int* n2;
    const gls_keypoint* k2;
};
struct MatchJobs {
    MatchJob j[kMaxJobs];
};

// matchKeyPoints (SURF.metal:441-487): the reference scans the train
// descriptors in 24 lanes, j = lane, lane + 24, ..., each keeping its first
// smallest distance, and takes the lanes in order, strictly smaller wins: the
// minimum over (distance, j mod 24, j). The distance is the square root of
// four float lane sums (SURF.metal:423-431), each in component order.
//
// Here a block of 256 threads takes 64 queries and a share of the train set,
// 64 at a time staged in shared memory, and a thread 4 x 4 pairs: every
// staged component serves four pairs from registers. Components travel as
// packed FP32 pairs (two lane sums an instruction; the train values are
// staged negated, q + (-t) rounds as q - t). The pair keys, distance bits
// over (j mod 24, j), are reduced by shuffles and one 64-bit atomic minimum
// per query and block, so the train set can be split over blocks. Bound by
// the FP32 pipe's subtract, multiply and add (the reference's roundings
// leave no FMA; 80% busy): 0.25 ms for 14 jobs of 1500 x 1500, 2.11 ms with a
// warp per query that read whole descriptors per lane.
typedef unsigned long long u64;
constexpr int MT = 64, MT_PAD = MT + 1;  // tile edge; padded so that staging stores and reads are conflict-free
constexpr u64 kOne2 = 0x3f8000003f800000ull;  // (1, 1)
constexpr u64 kNoMatch = ~0ull;          // no distance below FLT_MAX: reported as train 0 at FLT_MAX

struct MatchSmem {
    float4 q[16][MT_PAD], t[16][MT_PAD];  // component group, descriptor
};

__device__ __forceinline__ u64 add_f32x2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 mul_f32x2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 fma_f32x2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float2 unpack_f32x2(u64 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

// descriptors [first, first + 64) of n, negated if NEG, into a tile (zeros past n)
template <bool NEG>
__device__ __forceinline__ void stage_desc(float4 (*tile)[MT_PAD], const float* __restrict__ d, int first, int n) {
#pragma unroll
    for (int k = 0; k < MT * 16 / 256; k++) {
        const int e = threadIdx.x + 256 * k, row = e / 16, g = e % 16;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (first + row < n) v = __ldg(reinterpret_cast<const float4*>(d + size_t(first + row) * 64) + g);
        tile[g][row] = NEG ? make_float4(-v.x, -v.y, -v.z, -v.w) : v;
    }
}

__global__ void __launch_bounds__(256, 2) k_match(MatchJobs jobs, int cap, u64 one, u64* __restrict__ keys) {
    __shared__ MatchSmem sm;
    const MatchJob& J = jobs.j[blockIdx.y];
    const int n1 = *J.n1, n2 = *J.n2;
    const int q0 = blockIdx.x * MT;
    if (q0 >= n1) return;
    const int tiles = (n2 + MT - 1) / MT;
    const int t0 = int(int64_t(tiles) * blockIdx.z / gridDim.z), t1 = int(int64_t(tiles) * (blockIdx.z + 1) / gridDim.z);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    stage_desc<false>(sm.q, J.d1, q0, n1);
    u64 best[4] = {kNoMatch, kNoMatch, kNoMatch, kNoMatch};
    for (int tile = t0; tile < t1; tile++) {
        __syncthreads();  // the previous tile is read
        stage_desc<true>(sm.t, J.d2, tile * MT, n2);
        __syncthreads();
        u64 s01[4][4], s23[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s01[i][j] = s23[i][j] = 0;
#pragma unroll 2
        for (int g = 0; g < 16; g++) {
            ulonglong2 q[4];
#pragma unroll
            for (int i = 0; i < 4; i++) q[i] = *reinterpret_cast<const ulonglong2*>(&sm.q[g][ty + 16 * i]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&sm.t[g][tx + 16 * j]);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const u64 e01 = add_f32x2(q[i].x, t.x), e23 = add_f32x2(q[i].y, t.y);
                    // 1 x + s rounds as the sum; `one` comes from the launch,
                    // since a packed multiply and add, or a multiply-add by a
                    // known 1, is contracted into one rounding
                    s01[i][j] = fma_f32x2(mul_f32x2(e01, e01), one, s01[i][j]);
                    s23[i][j] = fma_f32x2(mul_f32x2(e23, e23), one, s23[i][j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int jt = tile * MT + tx + 16 * j;
            const unsigned low = (unsigned(jt % 24) << 27) | unsigned(jt);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a = unpack_f32x2(s01[i][j]), b = unpack_f32x2(s23[i][j]);
                const float d = fsqrt(fadd(fadd(fadd(a.x, a.y), b.x), b.y));
                if (jt < n2 && d < FLT_MAX) {
                    const u64 key = (u64(__float_as_uint(d)) << 32) | low;
                    best[i] = key < best[i] ? key : best[i];
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {  // over the 16 threads of a query
            const u64 v = __shfl_xor_sync(0xffffffffu, best[i], o);
            best[i] = v < best[i] ? v : best[i];
        }
        const int q = q0 + ty + 16 * i;
        if (tx == 0 && q < n1 && best[i] != kNoMatch) atomicMin(keys + size_t(blockIdx.y) * cap + q, best[i]);
    }
}

// refineMatch order (SURF.cpp:917-929): distance, then query index; the
// sorted matches become point pairs (query pt, train pt) as findMatches
// builds them (SURF.hpp:65-75). A block ranks 64 matches, four threads each
// scanning a quarter of the others ((distance bits, query index) as one
// 64-bit key: distances are not negative).
constexpr int MR_N = 64;
__global__ void __launch_bounds__(256) k_match_rank(MatchJobs jobs, int cap, const u64* __restrict__ keys_all,
                                                    gls_match* __restrict__ sorted_all, float4* __restrict__ pairs_all) {
    __shared__ u64 tile[1024];
    const MatchJob& J = jobs.j[blockIdx.y];
    const u64* __restrict__ keys = keys_all + size_t(blockIdx.y) * cap;
    gls_match* __restrict__ sorted = sorted_all + size_t(blockIdx.y) * cap;
    float4* __restrict__ pairs = pairs_all + size_t(blockIdx.y) * cap;
    const int n = *J.n1;
    const int i = blockIdx.x * MR_N + (threadIdx.x >> 2), part = threadIdx.x & 3;
    if (blockIdx.x * MR_N >= n) return;
    auto distance = [](u64 key) { return key == kNoMatch ? FLT_MAX : __uint_as_float(unsigned(key >> 32)); };
    auto rank_key = [&](u64 key, int q) { return (u64(__float_as_uint(distance(key))) << 32) | unsigned(q); };
    const u64 mine = i < n ? keys[i] : 0, me = rank_key(mine, i);
    int rank = 0;
    for (int j0 = 0; j0 < n; j0 += 1024) {
        __syncthreads();
        for (int j = threadIdx.x; j < 1024; j += 256) tile[j] = j0 + j < n ? rank_key(keys[j0 + j], j0 + j) : kNoMatch;
        __syncthreads();
        const int c = min(1024, n - j0);
#pragma unroll 8
        for (int j = part; j < c; j += 4) rank += tile[j] < me ? 1 : 0;
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    if (i < n && part == 0) {
        const int train = mine == kNoMatch ? 0 : int(mine & ((1u << 27) - 1));
        sorted[rank] = {i, train, distance(mine)};
        const gls_keypoint a = J.k1[i], b = J.k2[train];
        pairs[rank] = make_float4(a.x, a.y, b.x, b.y);
    }
}

// ------------------------------------------------------------ homography
// FindLeastSquaresHomography (LeastSquaresHomography.cpp:355-423) with the
// Jacobi solver of :218-353; hypot(p, q) is sqrt(p^2 + q^2). Every value is
// the sequential loop's, bit for bit: a Jacobi step's rotations update disjoint
// element pairs, and the scans for the next pivot compare the same values in
// an order whose result does not depend on it.
//
// Ten lanes solve one system, three systems to a warp (lanes 30 and 31 idle
// along with the third): lane r of a group owns row r. The pivot choice is a
// 9-lane tournament, the rotation parameters (two square roots, three
// divisions, most of a step's instructions) are formed by all lanes of the
// three groups at once, and lanes k and l rescan their rows together. A
// 4-point fit takes about 136 steps; a step costs a warp about 490 issue
// slots for three systems where a warp per system, with its serial scans on
// one lane, took about 660 for one: 2.16 -> 0.74 ms for 14 x 2000 fits (73%
// of the issue slots, FP64 pipe 34%).
__device__ __forceinline__ double hypot_d(double a, double b) { return dsqrt(dadd(dmul(a, a), dmul(b, b))); }

constexpr unsigned kFull = 0xffffffffu;
constexpr int LS_LANES = 10, LS_GROUPS = 3;

struct LsGroup {  // shared scratch of one system
    double a[9][10];        // the symmetric matrix, both triangles (destroyed)
    double V[9][9];         // eigenvectors as rows, in the order before sorting
    double T[9];
    double cen[4], mad[4];  // (cm0, cm1, cM0, cM1) and (sm0, sm1, sM0, sM1)
};

// a lane's place: its group's first lane and its row (9 and more: idle)
struct LsLane {
    int base, r;
};
__device__ __forceinline__ LsLane ls_lane() {
    const int lane = threadIdx.x & 31, g = min(lane / LS_LANES, LS_GROUPS - 1);
    return {g * LS_LANES, lane - g * LS_LANES};
}

__device__ __forceinline__ void jac_rot(double& v0, double& v1, double c, double s) {
    const double a0 = v0, b0 = v1;
    v0 = dsub(dmul(a0, c), dmul(b0, s));
    v1 = dadd(dmul(a0, s), dmul(b0, c));
}

// of row r of the symmetric matrix: the column right of the diagonal and the
// one left of it with the largest magnitude, the first on ties (indR, indC)
__device__ __forceinline__ void row_maxima(const double* row, int r, int& right, int& left) {
    double mr = 0.0, ml = 0.0;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const double v = fabs(row[j]);
        if (j > r && (j == r + 1 || mr < v)) mr = v, right = j;
        if (j < r && (j == 0 || ml < v)) ml = v, left = j;
    }
}

// Jacobi eigen-solve of the group's S.a: returns the row of S.V that the
// reference's sort (descending eigenvalues) puts last. Called by a whole
// warp; groups with run = false only take part in the shuffles.
__device__ int jacobi9(LsGroup& S, LsLane L, bool run) {
    constexpr int N = 9;
    const int r = L.r, row = min(r, N - 1);
    const bool lane_on = run && r < N;
    double* mine = S.a[row];
    double W = 0.0;
    int indR = N - 1, indC = 0;
    if (lane_on) {
#pragma unroll
        for (int i = 0; i < N; i++) S.V[row][i] = i == row ? 1.0 : 0.0;
        W = mine[row];
        row_maxima(mine, row, indR, indC);
    }
    __syncwarp();
    bool active = run;
    for (int it = 0; it < N * N * 30; it++) {
        // the pivot: the largest |a[i][indR[i]]| (i = 0..7), then
        // |a[indC[i]][i]| (i = 1..8), the first of equals; a NaN in the very
        // first place is kept, elsewhere it never wins
        double v = -1.0;
        int code = 31;
        if (lane_on && active) {
            if (r < N - 1) {
                v = fabs(mine[indR]);
                code = r;
                if (isnan(v)) v = r == 0 ? __longlong_as_double(0x7ff0000000000000ll) : -1.0;
            }
            if (r > 0) {
                const double vc = fabs(mine[indC]);
                if (v < vc) v = vc, code = 16 + r;
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const double ov = __shfl_down_sync(kFull, v, o);
            const int oc = __shfl_down_sync(kFull, code, o);
            if (r + o < N && r < o && (v < ov || (v == ov && oc < code))) v = ov, code = oc;
        }
        code = __shfl_sync(kFull, code, L.base) & 31;
        const int from = code & 15, ind = __shfl_sync(kFull, indR | (indC << 8), L.base + min(from, N - 1));
        int k = code < 16 ? from : ind >> 8, l = code < 16 ? ind & 255 : from;
        k = min(k, N - 1);
        l = min(l, N - 1);
        const double Wk = __shfl_sync(kFull, W, L.base + k), Wl = __shfl_sync(kFull, W, L.base + l);
        const double p = S.a[k][l];
        active = active && !(fabs(p) <= DBL_EPSILON);
        if (!__any_sync(kFull, active)) break;
        const double y = dmul(dsub(Wl, Wk), 0.5);
        double t = dadd(fabs(y), hypot_d(p, y));
        double s = hypot_d(p, t);
        const double c = ddiv(t, s);
        s = ddiv(p, s);
        t = dmul(ddiv(p, t), p);
        if (y < 0) {
            s = -s;
            t = -t;
        }
        __syncwarp();  // p is read by every lane
        if (lane_on && active) {
            if (r == k) {
                W = dsub(W, t);
                mine[l] = 0.0;
            } else if (r == l) {
                W = dadd(W, t);
                mine[k] = 0.0;
            } else {
                double ek = mine[k], el = mine[l];
                jac_rot(ek, el, c, s);
                mine[k] = ek;
                mine[l] = el;
                S.a[k][r] = ek;
                S.a[l][r] = el;
            }
            jac_rot(S.V[k][r], S.V[l][r], c, s);
        }
        __syncwarp();
        if (lane_on && active && (r == k || r == l)) row_maxima(mine, row, indR, indC);
    }
    // the selection sort of the eigenvalues, every lane of the group alike
    double w[N];
    int perm[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        w[i] = __shfl_sync(kFull, W, L.base + i);
        perm[i] = i;
    }
#pragma unroll
    for (int k = 0; k < N - 1; k++) {
        int m = k, pm = perm[k];
        double wm = w[k];
#pragma unroll
        for (int i = k + 1; i < N; i++)
            if (wm < w[i]) wm = w[i], pm = perm[i], m = i;
#pragma unroll
        for (int i = k + 1; i < N; i++)
            if (i == m) w[i] = w[k], perm[i] = perm[k];
        w[k] = wm;
        perm[k] = pm;
    }
    __syncwarp();
    return perm[N - 1];
}

// the rows Lx, Ly of LeastSquaresHomography.cpp:396-397 for a normalised
// point pair (a0, a1) -> (b0, b1)
__device__ __forceinline__ void ls_rows(double a0, double a1, double b0, double b1, double* lx, double* ly) {
    lx[0] = a0, lx[1] = a1, lx[2] = 1.0, lx[3] = lx[4] = lx[5] = 0.0;
    lx[6] = dmul(-b0, a0), lx[7] = dmul(-b0, a1), lx[8] = -b0;
    ly[0] = ly[1] = ly[2] = 0.0, ly[3] = a0, ly[4] = a1, ly[5] = 1.0;
    ly[6] = dmul(-b1, a0), ly[7] = dmul(-b1, a1), ly[8] = -b1;
}

// upper-triangle entry e (0..44) -> (j, k), j <= k
__device__ __forceinline__ void tri_index(int e, int& j, int& k) {
    j = 0;
    while (e >= 9 - j) {
        e -= 9 - j;
        j++;
    }
    k = j + e;
}

// The tail of the normalised DLT on S.a, S.cen and S.mad: least
// eigenvector, de-normalisation, scale to H[2][2] = 1. Warp.
__device__ void ls_finish(LsGroup& S, LsLane L, bool run, float* H) {
    const double* h0 = S.V[jacobi9(S, L, run)];
    const int r = min(L.r, 8), i = r / 3, j = r % 3;
    double q = 0.0;
    if (run) {
        const double cm0 = S.cen[0], cm1 = S.cen[1], sm0 = S.mad[0], sm1 = S.mad[1];
        const double inv[9] = {sm0, 0, cm0, 0, sm1, cm1, 0, 0, 1};
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double e = i == 0 ? inv[k] : i == 1 ? inv[3 + k] : inv[6 + k];
            acc = dadd(acc, dmul(e, h0[k * 3 + j]));
        }
        if (L.r < 9) S.T[r] = acc;
    }
    __syncwarp();
    if (run) {
        const double cM0 = S.cen[2], cM1 = S.cen[3], sM0 = S.mad[2], sM1 = S.mad[3];
        const double nrm[9] = {ddiv(1.0, sM0), 0, ddiv(-cM0, sM0), 0, ddiv(1.0, sM1), ddiv(-cM1, sM1), 0, 0, 1};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double e = j == 0 ? nrm[3 * k] : j == 1 ? nrm[3 * k + 1] : nrm[3 * k + 2];
            q = dadd(q, dmul(S.T[i * 3 + k], e));
        }
    }
    const double q8 = __shfl_sync(kFull, q, L.base + 8);
    if (run && L.r < 9) H[r] = fdiv(__double2float_rn(q), __double2float_rn(q8));
    __syncwarp();
}

// The 4-point models of the RANSAC samples idx of a warp's groups; a group
// whose spread is degenerate (where the reference throws) gets the identity.
__device__ void ls4(LsGroup& S, LsLane L, bool run, const float4* __restrict__ P, const int* __restrict__ idx,
                    float* H) {
    const int r = L.r;
    auto comp = [](const float4& p, int c) { return c == 0 ? p.z : c == 1 ? p.w : c == 2 ? p.x : p.y; };
    // the rows of the four points, in the place of V (built after them)
    double(*lx)[9] = S.V, (*ly)[9] = S.V + 4;
    if (run && r < 4) {
        double acc = 0.0;
        for (int i = 0; i < 4; i++) acc = dadd(acc, double(comp(P[idx[i]], r)));
        const double cen = ddiv(acc, 4.0);
        acc = 0.0;
        for (int i = 0; i < 4; i++) acc = dadd(acc, fabs(dsub(double(comp(P[idx[i]], r)), cen)));
        S.cen[r] = cen;
        S.mad[r] = ddiv(acc, 4.0);
    }
    __syncwarp();
    bool degenerate = false;
    if (run) {
        const double eps = DBL_EPSILON;
        degenerate =
            fabs(S.mad[0]) < eps || fabs(S.mad[1]) < eps || fabs(S.mad[2]) < eps || fabs(S.mad[3]) < eps;
    }
    const bool fit = run && !degenerate;
    if (fit && r < 4) {
        const float4 p = P[idx[r]];
        ls_rows(ddiv(dsub(double(p.x), S.cen[2]), S.mad[2]), ddiv(dsub(double(p.y), S.cen[3]), S.mad[3]),
                ddiv(dsub(double(p.z), S.cen[0]), S.mad[0]), ddiv(dsub(double(p.w), S.cen[1]), S.mad[1]), lx[r],
                ly[r]);
    }
    __syncwarp();
    if (fit && r < 9) {
        for (int e = r; e < 45; e += 9) {
            int j, k;
            tri_index(e, j, k);
            double acc = 0.0;
#pragma unroll
            for (int q = 0; q < 4; q++) acc = dadd(acc, dadd(dmul(lx[q][j], lx[q][k]), dmul(ly[q][j], ly[q][k])));
            S.a[j][k] = acc;
            S.a[k][j] = acc;  // completeSymm
        }
    }
    __syncwarp();
    ls_finish(S, L, fit, H);
    if (run && degenerate && r < 9) H[r] = (r % 4 == 0) ? 1.0f : 0.0f;
    __syncwarp();
}

// applyHomography + squared error (Homography.cpp:65-70)
__device__ __forceinline__ float h_error(const float* H, float4 p) {
    const float w = fadd(fadd(fmul(H[6], p.x), fmul(H[7], p.y)), H[8]);
    const float u = fdiv(fadd(fadd(fmul(H[0], p.x), fmul(H[1], p.y)), H[2]), w);
    const float v = fdiv(fadd(fadd(fmul(H[3], p.x), fmul(H[4], p.y)), H[5]), w);
    const float dx = fsub(u, p.z), dy = fsub(v, p.w);
    return fadd(fmul(dx, dx), fmul(dy, dy));
}

// One RANSAC problem per job: its point pairs, their count and the sample
// table drawn for that count.
struct RansacJob {
    const float4* pairs;
    const int* samples;
    int n;
};
struct RansacJobs {
    RansacJob j[kMaxJobs];
};

// RANSAC hypotheses (RTL/RANSAC.hpp:47-66, 101-108): a warp fits three
// iterations' samples and counts the errors above the threshold of the three
// models in one pass over the pairs.
constexpr int kHypWarps = 4, kHypModels = kHypWarps * LS_GROUPS;
__global__ void __launch_bounds__(32 * kHypWarps) k_ransac_models(RansacJobs jobs, int iters, float threshold,
                                                                  float* __restrict__ models_all,
                                                                  int* __restrict__ losses_all) {
    __shared__ LsGroup S[kHypWarps][LS_GROUPS];
    __shared__ float Hs[kHypWarps][LS_GROUPS][9];
    const RansacJob& J = jobs.j[blockIdx.y];
    const float4* __restrict__ pairs = J.pairs;
    const int n = J.n;
    float* __restrict__ models = models_all + size_t(blockIdx.y) * iters * 9;
    int* __restrict__ losses = losses_all + size_t(blockIdx.y) * iters;
    const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
    const LsLane L = ls_lane();
    const int g = L.base / LS_LANES, it0 = (blockIdx.x * kHypWarps + w) * LS_GROUPS, it = it0 + g;
    if (it0 >= iters) return;  // warp-uniform
    ls4(S[w][g], L, it < iters, pairs, J.samples + 4 * min(it, iters - 1), Hs[w][g]);
    const int ng = min(LS_GROUPS, iters - it0);
    float H[LS_GROUPS][9];
#pragma unroll
    for (int m = 0; m < LS_GROUPS; m++)
#pragma unroll
        for (int e = 0; e < 9; e++) H[m][e] = Hs[w][min(m, ng - 1)][e];
    int c[LS_GROUPS] = {0, 0, 0};
    for (int i = lane; i < n; i += 32) {
        const float4 p = pairs[i];
#pragma unroll
        for (int m = 0; m < LS_GROUPS; m++) c[m] += fabsf(h_error(H[m], p)) > threshold ? 1 : 0;
    }
#pragma unroll
    for (int m = 0; m < LS_GROUPS; m++) {
        for (int o = 16; o > 0; o >>= 1) c[m] += __shfl_xor_sync(kFull, c[m], o);
        if (m < ng && lane == 0) losses[it0 + m] = c[m];
    }
    for (int e = lane; e < 9 * ng; e += 32) models[it0 * 9 + e] = Hs[w][e / 9][e % 9];
}

// The first model with the least loss, its inliers (|error| < threshold,
// in index order) and, with 4 or more, their least-squares refit
// (Homography.cpp:90-113). One block a job: bound by the serial FP64 additions
// and the Jacobi steps; the terms of the sums are formed by all threads into
// shared memory, off the chains (0.70 -> 0.20 ms at about 1000 inliers).
constexpr int kFinalThreads = 256;
constexpr int kStage = 512, kRows = 32;  // inliers staged: for the sums, for the normal matrix
__global__ void __launch_bounds__(kFinalThreads) k_ransac_final(RansacJobs jobs, int cap,
                                                                 const float* __restrict__ models_all,
                                                                 const int* __restrict__ losses_all, int iters,
                                                                 float threshold, int* __restrict__ inliers_all,
                                                                 int* __restrict__ n_inliers_all,
                                                                 float* __restrict__ H_all,
                                                                 float* __restrict__ loss_all) {
    const int job = blockIdx.x;
    const float4* __restrict__ pairs = jobs.j[job].pairs;
    const int n = jobs.j[job].n;
    const float* __restrict__ models = models_all + size_t(job) * iters * 9;
    const int* __restrict__ losses = losses_all + size_t(job) * iters;
    int* __restrict__ inliers = inliers_all + size_t(job) * cap;
    int* __restrict__ n_inliers = n_inliers_all + job;
    float* __restrict__ Hout = H_all + size_t(job) * 9;
    float* __restrict__ loss_out = loss_all + job;
    __shared__ int best_s, base_s;
    __shared__ float H[9], Hf[9];
    __shared__ int wsum[kFinalThreads / 32];
    __shared__ LsGroup S[LS_GROUPS];  // the first is the refit's, the others idle along
    __shared__ double stage[4][kStage];
    __shared__ double lx[kRows][9], ly[kRows][9], prod[kRows][45];
    __shared__ int red_loss[kFinalThreads / 32], red_idx[kFinalThreads / 32];
    __shared__ int tri[45];  // upper-triangle entry -> 9 j + k
    const int t = threadIdx.x;
    if (t < 45) {
        int j, k;
        tri_index(t, j, k);
        tri[t] = 9 * j + k;
    }
    {  // the first iteration with the least loss: (loss, index) minimum
        int bl = INT_MAX, bi = INT_MAX;
        for (int i = t; i < iters; i += kFinalThreads) {
            const int v = losses[i];
            if (v < bl) bl = v, bi = i;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const int ol = __shfl_xor_sync(kFull, bl, o), oi = __shfl_xor_sync(kFull, bi, o);
            if (ol < bl || (ol == bl && oi < bi)) bl = ol, bi = oi;
        }
        if ((t & 31) == 0) {
            red_loss[t >> 5] = bl;
            red_idx[t >> 5] = bi;
        }
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < kFinalThreads / 32; w++)
                if (red_loss[w] < bl || (red_loss[w] == bl && red_idx[w] < bi)) bl = red_loss[w], bi = red_idx[w];
            best_s = bi;
            base_s = 0;
        }
    }
    __syncthreads();
    if (t < 9) H[t] = models[best_s * 9 + t];
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += kFinalThreads) {  // ordered compaction of the inliers
        const int i = i0 + t;
        const int f = (i < n && fabsf(h_error(H, pairs[i])) < threshold) ? 1 : 0;
        const unsigned bal = __ballot_sync(kFull, f);
        const int lane = t & 31, w = t >> 5;
        if (lane == 0) wsum[w] = __popc(bal);
        __syncthreads();
        int off = base_s;
        for (int k = 0; k < w; k++) off += wsum[k];
        if (f) inliers[off + __popc(bal & ((1u << lane) - 1u))] = i;
        __syncthreads();
        if (t == 0) {
            int s = 0;
            for (int k = 0; k < kFinalThreads / 32; k++) s += wsum[k];
            base_s += s;
        }
        __syncthreads();
    }
    const int m = base_s;
    if (t == 0) {
        *n_inliers = m;
        *loss_out = float(losses[best_s]);
    }
    auto comp = [](const float4& p, int c) { return c == 0 ? p.z : c == 1 ? p.w : c == 2 ? p.x : p.y; };
    bool refit = false;
    if (m >= 4) {
        // centroids, then mean absolute deviations: sequential sums over the
        // inliers in index order, a thread per component; the terms are formed
        // by all threads, so the serial path is one FP64 addition an inlier
        for (int pass = 0; pass < 2; pass++) {
            double acc = 0.0;
            for (int c0 = 0; c0 < m; c0 += kStage) {
                const int cnt = min(kStage, m - c0);
                __syncthreads();
                for (int i = t; i < cnt; i += kFinalThreads) {
                    const float4 p = pairs[inliers[c0 + i]];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const double v = double(comp(p, c));
                        stage[c][i] = pass == 0 ? v : fabs(dsub(v, S[0].cen[c]));
                    }
                }
                __syncthreads();
                if (t < 4) {
                    int i = 0;
                    for (; i + 16 <= cnt; i += 16) {
#pragma unroll
                        for (int u = 0; u < 16; u++) acc = dadd(acc, stage[t][i + u]);
                    }
                    for (; i < cnt; i++) acc = dadd(acc, stage[t][i]);
                }
            }
            if (t < 4) {
                if (pass == 0) S[0].cen[t] = ddiv(acc, double(m));
                else S[0].mad[t] = ddiv(acc, double(m));
            }
            __syncthreads();
        }
        const double eps = DBL_EPSILON;
        const bool degenerate =
            fabs(S[0].mad[0]) < eps || fabs(S[0].mad[1]) < eps || fabs(S[0].mad[2]) < eps || fabs(S[0].mad[3]) < eps;
        if (!degenerate) {
            // the normal matrix, entry by entry in inlier order: a thread per
            // inlier forms its rows, all threads the 45 products of each
            // inlier, and 45 threads add them up, one FP64 addition an inlier
            // on the serial path
            double acc = 0.0;
            for (int c0 = 0; c0 < m; c0 += kRows) {
                const int cnt = min(kRows, m - c0);
                __syncthreads();
                for (int i = t; i < cnt; i += kFinalThreads) {
                    const float4 p = pairs[inliers[c0 + i]];
                    ls_rows(ddiv(dsub(double(p.x), S[0].cen[2]), S[0].mad[2]),
                            ddiv(dsub(double(p.y), S[0].cen[3]), S[0].mad[3]),
                            ddiv(dsub(double(p.z), S[0].cen[0]), S[0].mad[0]),
                            ddiv(dsub(double(p.w), S[0].cen[1]), S[0].mad[1]), lx[i], ly[i]);
                }
                __syncthreads();
                for (int e = t; e < cnt * 45; e += kFinalThreads) {
                    const int i = e / 45;
                    const int jk = tri[e % 45], j = jk / 9, k = jk % 9;
                    prod[i][e % 45] = dadd(dmul(lx[i][j], lx[i][k]), dmul(ly[i][j], ly[i][k]));
                }
                __syncthreads();
                if (t < 45) {
                    if (cnt == kRows) {
#pragma unroll
                        for (int i = 0; i < kRows; i++) acc = dadd(acc, prod[i][t]);
                    } else {
                        for (int i = 0; i < cnt; i++) acc = dadd(acc, prod[i][t]);
                    }
                }
            }
            if (t < 45) {
                const int j = tri[t] / 9, k = tri[t] % 9;
                S[0].a[j][k] = acc;
                S[0].a[k][j] = acc;  // completeSymm
            }
            __syncthreads();
            if (t < 32) {
                const LsLane L = ls_lane();
                ls_finish(S[L.base / LS_LANES], L, L.base == 0, Hf);
            }
            refit = true;
            __syncthreads();
        }
    }
    if (t < 9) Hout[t] = refit ? Hf[t] : H[t];
}

// ------------------------------------------------------------ raw channels
struct ChanArgs {
    const uint16_t* raw;
    size_t stride;  // elements
    int ow, oh;
    int ox[4], oy[4];
    float* out[4];
    int out_pitch[4];  // floats
    uint32_t mask;
    const float* lut;
};

// RawChannels (pyramidFusion.cpp:132-139) through a 65536-entry tone-curve
// table built on the host with the reference's expression.
__global__ void k_raw_channels(ChanArgs a) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= a.ow || y >= a.oh) return;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        if (!(a.mask & (1u << c))) continue;
        const uint16_t v = __ldg(a.raw + size_t(2 * y + a.oy[c]) * a.stride + 2 * x + a.ox[c]);
        a.out[c][size_t(y) * a.out_pitch[c] + x] = __ldg(a.lut + v);
    }
}

// ------------------------------------------------------------ integral
constexpr int IT = 32;  // integral tile edge
constexpr int IM = 8;   // warps that move a tile's values
constexpr int ID = 8;   // tiles loaded ahead

// A strip of 32 running sums, tile by tile: one warp adds down the tile's 32
// rows (a lane a sum, sequential in float) while the others write the tile
// before it, put the next one into shared memory and load the one after the
// next two: one barrier a tile, three tile buffers. Bound by the serial
// additions and the scan warp's way through shared memory; only W / 32 or H / 32
// blocks have work. 2016x1512: columns 33 us, rows 40 (38 and 48 with three
// barriers a tile, the scan between them).
// load(tile, k): value of row k of the tile for this lane; out(tile, k, buffer).
template <class Load, class Out>
__device__ __forceinline__ void running_sums(int tiles, float sub, Load load, Out out) {
    __shared__ float buf[3][IT][IT + 1];
    const int lane = threadIdx.x, w = threadIdx.y;
    float acc = 0.0f, next[ID][IT / IM];
    auto fetch = [&](int t, float (&v)[IT / IM]) {
#pragma unroll
        for (int k = 0; k < IT / IM; k++) v[k] = load(t, w + IM * k);
    };
    auto put = [&](int t, const float (&v)[IT / IM]) {
#pragma unroll
        for (int k = 0; k < IT / IM; k++) buf[t % 3][w + IM * k][lane] = v[k];
    };
    auto flush = [&](int t) {
#pragma unroll
        for (int k = 0; k < IT / IM; k++) out(t, w + IM * k, buf[t % 3]);
    };
    if (w < IM) {
#pragma unroll
        for (int t = 0; t < ID; t++) fetch(t, next[t]);
        put(0, next[0]);
        fetch(ID, next[0]);
    }
    __syncthreads();
    auto step = [&](int t, float (&v)[IT / IM]) {  // v: tile t + 1
        if (w == IM) {
            float(&b)[IT][IT + 1] = buf[t % 3];
            float c[IT];
#pragma unroll
            for (int k = 0; k < IT; k++) c[k] = b[k][lane];
#pragma unroll
            for (int k = 0; k < IT; k++) c[k] = acc = fadd(acc, fsub(c[k], sub));
#pragma unroll
            for (int k = 0; k < IT; k++) b[k][lane] = c[k];
        } else {
            if (t > 0) flush(t - 1);
            put(t + 1, v);
            fetch(t + 1 + ID, v);
        }
        __syncthreads();
    };
    for (int t = 0; t < tiles; t += ID)
#pragma unroll
        for (int k = 0; k < ID; k++)
            if (t + k < tiles) step(t + k, next[(k + 1) % ID]);
    if (w < IM) flush(tiles - 1);
}

// Column pass (integral_sum_cols_image, SURF.metal:315-338): a running sum
// of (v - 0.5) down each column, written transposed (T[x][y]).
__global__ void __launch_bounds__(32 * (IM + 1)) k_integral_cols(const float* __restrict__ img, int pitch, int W, int H,
                                                                 float* __restrict__ T, int tpitch) {
    const int x0 = blockIdx.x * IT, lane = threadIdx.x;
    running_sums(
        (H + IT - 1) / IT, 0.5f,
        [&](int t, int r) {
            const int x = x0 + lane, y = t * IT + r;
            return x < W && y < H ? __ldg(img + size_t(y) * pitch + x) : 0.0f;
        },
        [&](int t, int c, const float (&b)[IT][IT + 1]) {
            const int x = x0 + c, y = t * IT + lane;
            if (x < W && y < H) T[size_t(x) * tpitch + y] = b[lane][c];
        });
}

// Row pass (integral_sum_rows_image, SURF.metal:340-421): a running sum of
// the column sums along each row into the (W+1) x (H+1) sum image with a zero
// first row and column.
__global__ void __launch_bounds__(32 * (IM + 1)) k_integral_rows(const float* __restrict__ T, int tpitch, int W, int H,
                                                                 float* __restrict__ S, int spitch) {
    const int y0 = blockIdx.x * IT, lane = threadIdx.x;
    if (blockIdx.x == 0)
        for (int x = threadIdx.y * IT + lane; x <= W; x += (IM + 1) * IT) S[x] = 0.0f;
    if (threadIdx.y == 0 && y0 + lane < H) S[size_t(y0 + lane + 1) * spitch] = 0.0f;
    running_sums(
        (W + IT - 1) / IT, 0.0f,
        [&](int t, int c) {
            const int x = t * IT + c, y = y0 + lane;
            return x < W && y < H ? __ldg(T + size_t(x) * tpitch + y) : 0.0f;
        },
        [&](int t, int r, const float (&b)[IT][IT + 1]) {
            const int x = t * IT + lane, y = y0 + r;
            if (x < W && y < H) S[size_t(y + 1) * spitch + x + 1] = b[lane][r];
        });
}

// ------------------------------------------------------------ warps
struct WarpArgs {
    const float* fused;
    int fused_pitch;  // floats
    const void* input;
    int in_pitch;  // elements
    int iw, ih;
    float* out;
    int out_pitch;
    int w, h;
    float H[9];
    int count;  // 0: registerImage
};

// registerAndFuse / registerImage (SURF.metal:489-538): pull-warp by H with
// exact bilinear sampling, clamp-to-edge, and the running mean.
template <class S>
__global__ void __launch_bounds__(256) k_register(WarpArgs a) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= a.w || y >= a.h) return;
    float4 s = warp_sample(reinterpret_cast<const S*>(a.input), a.in_pitch, warp_pos(a.H, x, y, a.iw, a.ih));
    float4* o = reinterpret_cast<float4*>(a.out + size_t(y) * a.out_pitch + 4 * x);
    if (a.count > 0) {
        const float4 f = *reinterpret_cast<const float4*>(a.fused + size_t(y) * a.fused_pitch + 4 * x);
        const float cm1 = float(a.count - 1), cn = float(a.count);
        s = make_float4(fdiv(fadd(fmul(cm1, f.x), s.x), cn), fdiv(fadd(fmul(cm1, f.y), s.y), cn),
                        fdiv(fadd(fmul(cm1, f.z), s.z), cn), fdiv(fadd(fmul(cm1, f.w), s.w), cn));
    }
    *o = s;
}

}  // namespace gls

namespace gls {
struct FusionScratch;
FusionScratch* fusion_scratch_new();
void fusion_scratch_delete(FusionScratch* f);
gls_status fuse_pyramid_impl(FusionScratch* F, const gls_image_view* frames, int n, const float* H, int levels,
                             float robustness, gls_image_view* out, cudaStream_t s);
}  // namespace gls

// ============================================================ host object
using namespace gls;

struct SurfSlotState {
    DevBuf kps, desc, count;
    int count_host = -1;  // -1: not read back since the last detection
    bool valid = false;
};

struct gls_surf {
    int device = 0, W = 0, H = 0, max_features = 1500, n_oct = 4, n_layers = 2;
    float threshold = 0.02f;
    int capacity = 1500;  // keypoints kept per slot
    DevBuf img, sum, colT, cand, cand_count, tables;
    SurfSlotState slot[GLS_SURF_SLOTS];
    DevBuf matches, matches_sorted, pairs;  // [jobs][pair_cap]
    int pair_cap = 0;
    int match_query = -1, match_train = -1;  // the slots of the last single match (job 0)
    std::map<std::pair<int, int>, DevBuf> sample_tables;
    DevBuf models, losses, inliers, n_inliers, Hdev, loss;
    DevBuf raw, lut;
    float lut_black = NAN, lut_white = NAN, lut_exp = NAN;
    std::vector<float> lut_host;
    FusionScratch* fusion = nullptr;
    uint64_t launches = 0;
};

namespace {

gls_status check_surf(gls_surf* s) {
    if (!s) return set_error(GLS_ERR_INVALID_ARG, "NULL detector");
    GLS_CUDA(cudaSetDevice(s->device));
    return GLS_OK;
}

gls_status launch_check(gls_surf* s, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(GLS_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
    s->launches++;
    return GLS_OK;
}

// getGaussianKernel (SURF.cpp:394-425) for sigma > 0
std::vector<float> gaussian_kernel(int n, float sigma) {
    const float scale2X = float(-0.5 / double(sigma * sigma));
    float sum = 0;
    std::vector<float> k(n);
    for (int i = 0; i < n; i++) {
        const float x = float(i - (n - 1) * 0.5);
        k[i] = std::exp(scale2X * x * x);
        sum += k[i];
    }
    sum = float(1. / sum);
    for (auto& v : k) v *= sum;
    return k;
}

DescTables make_tables() {
    DescTables t{};
    const auto g = gaussian_kernel(13, 2.5f);
    for (int i = -6; i <= 6; i++)
        for (int j = -6; j <= 6; j++)
            if (i * i + j * j <= 36) {
                t.apt_x[t.n_ori] = float(i);
                t.apt_y[t.n_ori] = float(j);
                t.aptw[t.n_ori++] = g[i + 6] * g[j + 6];
            }
    const auto gd = gaussian_kernel(20, 3.3f);
    for (int i = 0; i < 20; i++)
        for (int j = 0; j < 20; j++) t.dw[i * 20 + j] = gd[i] * gd[j];
    return t;
}

// toneCurve / sigmoid (pyramidFusion.cpp:92-104) in the reference's mix of
// float and double.
float sigmoid(float x, float s) { return float(0.5 * (std::tanh(double(s * x) - 0.3 * s) + 1)); }
float tone_curve(float x, float s) {
    const float p = float(std::pow(0.95 * x, 0.5));
    return (sigmoid(p, s) - sigmoid(0.0f, s)) / (sigmoid(1.0f, s) - sigmoid(0.0f, s));
}

// mt19937 (default seed) with a mask-and-reject uniform integer in [0, n-1]:
// the 4-index sets of RTL::RANSAC::GenerateModel (RTL/RANSAC.hpp:95-99), each
// in ascending order.
std::vector<int> ransac_samples(int iterations, int n) {
    std::mt19937 g;
    const uint32_t range = uint32_t(n);
    int w = 0;
    while (w < 32 && (uint64_t(1) << w) < range) w++;
    const uint32_t mask = w >= 32 ? 0xffffffffu : ((1u << w) - 1u);
    std::vector<int> out(size_t(iterations) * 4);
    for (int it = 0; it < iterations; it++) {
        std::set<int> s;
        while (s.size() < 4) {
            int v = 0;
            if (range > 1) {
                uint32_t u;
                do {
                    u = uint32_t(g()) & mask;
                } while (u >= range);
                v = int(u);
            }
            s.insert(v);
            if (range < 4 && s.size() == range) break;
        }
        int k = 0;
        for (int v : s) out[size_t(it) * 4 + k++] = v;
        for (; k < 4; k++) out[size_t(it) * 4 + k] = *s.begin();
    }
    return out;
}

// the RANSAC sample table for n pairs (cached per (n, iterations))
gls_status sample_table(gls_surf* s, int n, int iters, const int** out, cudaStream_t st) {
    auto key = std::make_pair(n, iters);
    auto it = s->sample_tables.find(key);
    if (it == s->sample_tables.end()) {
        const std::vector<int> smp = ransac_samples(iters, n);
        DevBuf b;
        GLS_TRY(b.ensure(smp.size() * sizeof(int)));
        GLS_CUDA(cudaMemcpyAsync(b.p, smp.data(), smp.size() * sizeof(int), cudaMemcpyHostToDevice, st));
        GLS_CUDA(cudaStreamSynchronize(st));
        it = s->sample_tables.emplace(key, b).first;
    }
    *out = reinterpret_cast<const int*>(it->second.p);
    return GLS_OK;
}

// RANSAC + refit for jobs 0..J-1 whose pairs are in s->pairs (cap per job)
// and whose pair counts are ns[j]; leaves H [J][9], inliers, counts on the
// device.
gls_status run_ransac(gls_surf* s, const std::vector<int>& ns, float threshold, int iters, cudaStream_t st) {
    const int J = int(ns.size());
    const size_t cap = size_t(std::max(s->pair_cap, 1));
    RansacJobs rj{};
    for (int j = 0; j < J; j++) {
        if (ns[j] < 4) return set_error(GLS_ERR_DEGENERATE, "RANSAC needs at least 4 point pairs, got %d", ns[j]);
        rj.j[j].pairs = reinterpret_cast<const float4*>(s->pairs.p) + size_t(j) * cap;
        rj.j[j].n = ns[j];
        GLS_TRY(sample_table(s, ns[j], iters, &rj.j[j].samples, st));
    }
    GLS_TRY(s->models.ensure(size_t(J) * iters * 9 * sizeof(float)));
    GLS_TRY(s->losses.ensure(size_t(J) * iters * sizeof(int)));
    GLS_TRY(s->inliers.ensure(size_t(J) * cap * sizeof(int)));
    GLS_TRY(s->n_inliers.ensure(size_t(J) * sizeof(int)));
    GLS_TRY(s->Hdev.ensure(size_t(J) * 9 * sizeof(float)));
    GLS_TRY(s->loss.ensure(size_t(J) * sizeof(float)));
    k_ransac_models<<<dim3((iters + kHypModels - 1) / kHypModels, J), 32 * kHypWarps, 0, st>>>(
        rj, iters, threshold, reinterpret_cast<float*>(s->models.p), reinterpret_cast<int*>(s->losses.p));
    GLS_TRY(launch_check(s, "k_ransac_models"));
    k_ransac_final<<<J, kFinalThreads, 0, st>>>(rj, int(cap), reinterpret_cast<const float*>(s->models.p),
                                                reinterpret_cast<const int*>(s->losses.p), iters, threshold,
                                                reinterpret_cast<int*>(s->inliers.p),
                                                reinterpret_cast<int*>(s->n_inliers.p),
                                                reinterpret_cast<float*>(s->Hdev.p), reinterpret_cast<float*>(s->loss.p));
    GLS_TRY(launch_check(s, "k_ransac_final"));
    return GLS_OK;
}

// copies job 0's homography and inliers to the host (synchronising)
gls_status ransac_result(gls_surf* s, float* H, int32_t* inliers, int32_t* n_inl, cudaStream_t st) {
    int ni = 0;
    GLS_CUDA(cudaMemcpyAsync(H, s->Hdev.p, 9 * sizeof(float), cudaMemcpyDeviceToHost, st));
    GLS_CUDA(cudaMemcpyAsync(&ni, s->n_inliers.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    GLS_CUDA(cudaStreamSynchronize(st));
    if (n_inl) *n_inl = ni;
    if (inliers && ni > 0)
        GLS_CUDA(cudaMemcpy(inliers, s->inliers.p, size_t(ni) * sizeof(int), cudaMemcpyDeviceToHost));
    return GLS_OK;
}

gls_status ensure_pairs(gls_surf* s, int jobs, int cap) {
    s->pair_cap = std::max(s->pair_cap, cap);
    const size_t c = size_t(std::max(s->pair_cap, 1));
    GLS_TRY(s->matches.ensure(size_t(jobs) * c * sizeof(u64)));
    GLS_TRY(s->matches_sorted.ensure(size_t(jobs) * c * sizeof(gls_match)));
    GLS_TRY(s->pairs.ensure(size_t(jobs) * c * sizeof(float4)));
    return GLS_OK;
}

// match jobs (query slot, train slot) into matches / pairs job by job
gls_status run_match(gls_surf* s, const std::vector<std::pair<int, int>>& qt, cudaStream_t st) {
    const int J = int(qt.size());
    if (s->pair_cap != s->capacity) s->pair_cap = 0;
    GLS_TRY(ensure_pairs(s, J, s->capacity));
    MatchJobs mj{};
    for (int j = 0; j < J; j++) {
        const SurfSlotState &q = s->slot[qt[j].first], &t = s->slot[qt[j].second];
        mj.j[j] = {reinterpret_cast<const float*>(q.desc.p), reinterpret_cast<const int*>(q.count.p),
                   reinterpret_cast<const gls_keypoint*>(q.kps.p), reinterpret_cast<const float*>(t.desc.p),
                   reinterpret_cast<const int*>(t.count.p), reinterpret_cast<const gls_keypoint*>(t.kps.p)};
    }
    const int cap = s->pair_cap;
    u64* keys = reinterpret_cast<u64*>(s->matches.p);
    GLS_CUDA(cudaMemsetAsync(keys, 0xff, size_t(J) * cap * sizeof(u64), st));
    // the train set split so that the blocks of full slots fill about eight rounds
    // of two per SM (148): the last round's idle share stays near a tenth. The counts
    // are on the device: blocks past a slot's features leave at once (1076 by 1053
    // features in slots of 64000: registration 0.54 ms, 0.87 in its former form)
    const int tiles = (s->capacity + MT - 1) / MT;
    const int split = std::clamp(8 * 296 / std::max(tiles * J, 1), 1, std::max(tiles, 1));
    k_match<<<dim3(tiles, J, split), 256, 0, st>>>(mj, cap, kOne2, keys);
    GLS_TRY(launch_check(s, "k_match"));
    k_match_rank<<<dim3((s->capacity + MR_N - 1) / MR_N, J), 256, 0, st>>>(
        mj, cap, keys, reinterpret_cast<gls_match*>(s->matches_sorted.p), reinterpret_cast<float4*>(s->pairs.p));
    GLS_TRY(launch_check(s, "k_match_rank"));
    return GLS_OK;
}

}  // namespace

extern "C" {

gls_status gls_surf_create(int32_t device, int32_t width, int32_t height, int32_t max_features, int32_t n_octaves,
                           int32_t n_octave_layers, float hessian_threshold, gls_surf** out) {
    clear_error();
    if (!out) return set_error(GLS_ERR_INVALID_ARG, "NULL output");
    *out = nullptr;
    if (width < 1 || height < 1 || width > 32768 || height > 32768)
        return set_error(GLS_ERR_INVALID_ARG, "image size %dx%d out of range", width, height);
    if (n_octaves < 1 || n_octaves > kMaxOctaves)
        return set_error(GLS_ERR_INVALID_ARG, "n_octaves must be 1..%d", kMaxOctaves);
    if (n_octave_layers != 2)
        return set_error(GLS_ERR_UNSUPPORTED, "only 2 layers per octave (the reference's setting) are served");
    GLS_CUDA(cudaSetDevice(device));
    auto* s = new gls_surf();
    s->device = device;
    s->W = width;
    s->H = height;
    s->max_features = max_features;
    s->n_oct = n_octaves;
    s->n_layers = n_octave_layers;
    s->threshold = hessian_threshold;
    s->capacity = max_features < 0 ? kMaxKeypoints : std::min(max_features, kMaxKeypoints);
    auto fail = [&](gls_status st) {
        gls_surf_destroy(s);
        return st;
    };
    const size_t n = size_t(width) * height;
    gls_status st;
    if ((st = s->img.ensure(n * sizeof(float))) != GLS_OK) return fail(st);
    if ((st = s->sum.ensure(size_t(width + 1) * (height + 1) * sizeof(float))) != GLS_OK) return fail(st);
    if ((st = s->colT.ensure(n * sizeof(float))) != GLS_OK) return fail(st);
    if ((st = s->cand.ensure(size_t(kMaxKeypoints) * sizeof(gls_keypoint))) != GLS_OK) return fail(st);
    if ((st = s->cand_count.ensure(sizeof(int))) != GLS_OK) return fail(st);
    if ((st = s->tables.ensure(sizeof(DescTables))) != GLS_OK) return fail(st);
    const DescTables t = make_tables();
    if (cudaMemcpy(s->tables.p, &t, sizeof(t), cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(set_error(GLS_ERR_CUDA, "upload of the descriptor tables failed"));
    for (auto& sl : s->slot) {
        if ((st = sl.kps.ensure(size_t(std::max(s->capacity, 1)) * sizeof(gls_keypoint))) != GLS_OK) return fail(st);
        if ((st = sl.desc.ensure(size_t(std::max(s->capacity, 1)) * 64 * sizeof(float))) != GLS_OK) return fail(st);
        if ((st = sl.count.ensure(sizeof(int))) != GLS_OK) return fail(st);
        if (cudaMemset(sl.count.p, 0, sizeof(int)) != cudaSuccess)
            return fail(set_error(GLS_ERR_CUDA, "cudaMemset failed"));
    }
    *out = s;
    return GLS_OK;
}

gls_status gls_surf_destroy(gls_surf* s) {
    if (!s) return GLS_OK;
    cudaSetDevice(s->device);
    for (DevBuf* b : {&s->img, &s->sum, &s->colT, &s->cand, &s->cand_count, &s->tables, &s->matches,
                      &s->matches_sorted, &s->pairs, &s->models, &s->losses, &s->inliers, &s->n_inliers, &s->Hdev,
                      &s->loss, &s->raw, &s->lut})
        b->release();
    for (auto& kv : s->sample_tables) kv.second.release();
    if (s->fusion) fusion_scratch_delete(s->fusion);
    for (auto& sl : s->slot) {
        sl.kps.release();
        sl.desc.release();
        sl.count.release();
    }
    delete s;
    return GLS_OK;
}

gls_status gls_surf_detect_and_compute(gls_surf* s, const gls_image_view* img, int32_t slot, uint32_t flags,
                                       void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (!img || !img->data) return set_error(GLS_ERR_INVALID_ARG, "NULL image");
    if (slot < 0 || slot >= GLS_SURF_SLOTS) return set_error(GLS_ERR_INVALID_ARG, "slot %d out of range", slot);
    if (img->channels != 1 || img->dtype != GLS_F32)
        return set_error(GLS_ERR_INVALID_ARG, "image must be single-channel GLS_F32");
    if (img->width != s->W || img->height != s->H)
        return set_error(GLS_ERR_INVALID_ARG, "image is %dx%d, detector serves %dx%d", img->width, img->height, s->W,
                         s->H);
    const size_t stride = img->stride_bytes ? img->stride_bytes : size_t(img->width) * 4;
    if (stride % 4 || stride < size_t(img->width) * 4) return set_error(GLS_ERR_INVALID_ARG, "bad image stride");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const float* src = reinterpret_cast<const float*>(img->data);
    int pitch = int(stride / 4);
    if (flags & GLS_HOST_IO) {
        GLS_CUDA(cudaMemcpy2DAsync(s->img.p, size_t(s->W) * 4, img->data, stride, size_t(s->W) * 4, s->H,
                                   cudaMemcpyHostToDevice, st));
        src = reinterpret_cast<const float*>(s->img.p);
        pitch = s->W;
    }
    const int W = s->W, H = s->H;
    float* T = reinterpret_cast<float*>(s->colT.p);
    float* S = reinterpret_cast<float*>(s->sum.p);
    k_integral_cols<<<(W + IT - 1) / IT, dim3(32, IM + 1), 0, st>>>(src, pitch, W, H, T, H);
    GLS_TRY(launch_check(s, "k_integral_cols"));
    k_integral_rows<<<(H + IT - 1) / IT, dim3(32, IM + 1), 0, st>>>(T, H, W, H, S, W + 1);
    GLS_TRY(launch_check(s, "k_integral_rows"));
    // fastHessianDetector (SURF.cpp:1229-1286)
    DetectArgs da{};
    da.n_oct = s->n_oct;
    da.sum = S;
    da.sum_pitch = W + 1;
    da.sum_w = W + 1;
    da.sum_h = H + 1;
    da.threshold = s->threshold;
    da.per_axis = (flags & GLS_SURF_CORRECTED) ? 1 : 0;
    da.cand = reinterpret_cast<gls_keypoint*>(s->cand.p);
    da.cand_count = reinterpret_cast<int*>(s->cand_count.p);
    int blocks = 0;
    for (int o = 0; o < s->n_oct; o++) {
        OctaveDev& O = da.oct[o];
        O.step = 1 << o;
        for (int l = 0; l < kLayers; l++) O.layer[l] = make_layer(W + 1, H + 1, (9 + 6 * l) << o, O.step);
        O.lw = W / O.step;
        O.lh = H / O.step;
        O.tiles_x = std::max(1, (O.lw + DT_X - 1) / DT_X);
        O.tiles_y = std::max(1, (O.lh + DT_Y - 1) / DT_Y);
        O.block0 = blocks;
        blocks += O.tiles_x * O.tiles_y;
    }
    GLS_CUDA(cudaMemsetAsync(s->cand_count.p, 0, sizeof(int), st));
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_hessian_nms), int(sizeof(DetectSmem)));
    k_hessian_nms<<<blocks, 256, sizeof(DetectSmem), st>>>(da);
    GLS_TRY(launch_check(s, "k_hessian_nms"));
    SurfSlotState& sl = s->slot[slot];
    const int keep = s->capacity;
    k_keypoint_rank<<<(kMaxKeypoints + kRankPer - 1) / kRankPer, kRankPer * kRankLanes, 0, st>>>(
        reinterpret_cast<const gls_keypoint*>(s->cand.p), reinterpret_cast<const int*>(s->cand_count.p), keep,
        reinterpret_cast<gls_keypoint*>(sl.kps.p), reinterpret_cast<int*>(sl.count.p));
    GLS_TRY(launch_check(s, "k_keypoint_rank"));
    DescArgs ga{};
    ga.img = src;
    ga.img_pitch = pitch;
    ga.iw = W;
    ga.ih = H;
    ga.sum = S;
    ga.sum_pitch = W + 1;
    ga.sw = W + 1;
    ga.sh = H + 1;
    ga.tab = reinterpret_cast<const DescTables*>(s->tables.p);
    ga.kps = reinterpret_cast<gls_keypoint*>(sl.kps.p);
    ga.count = reinterpret_cast<const int*>(sl.count.p);
    ga.desc = reinterpret_cast<float*>(sl.desc.p);
    ga.all = (flags & GLS_SURF_CORRECTED) ? 1 : 0;
    if (keep > 0) {
        k_describe<<<keep, kDescThreads, 0, st>>>(ga);
        GLS_TRY(launch_check(s, "k_describe"));
    }
    sl.count_host = -1;
    sl.valid = true;
    if (s->match_query == slot || s->match_train == slot) s->match_query = s->match_train = -1;
    if (flags & (GLS_SYNC | GLS_HOST_IO)) GLS_CUDA(cudaStreamSynchronize(st));
    return GLS_OK;
}

static gls_status slot_count(gls_surf* s, int slot, cudaStream_t st, int* n) {
    SurfSlotState& sl = s->slot[slot];
    if (!sl.valid) return set_error(GLS_ERR_INVALID_ARG, "slot %d holds no detection", slot);
    if (sl.count_host < 0) {
        int c = 0;
        GLS_CUDA(cudaMemcpyAsync(&c, sl.count.p, sizeof(int), cudaMemcpyDeviceToHost, st));
        GLS_CUDA(cudaStreamSynchronize(st));
        sl.count_host = c;
    }
    *n = sl.count_host;
    return GLS_OK;
}

gls_status gls_surf_features(gls_surf* s, int32_t slot, gls_keypoint* kps, float* desc, int32_t capacity, int32_t* n,
                             void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (slot < 0 || slot >= GLS_SURF_SLOTS) return set_error(GLS_ERR_INVALID_ARG, "slot %d out of range", slot);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int c = 0;
    GLS_TRY(slot_count(s, slot, st, &c));
    if (n) *n = c;
    const int m = std::min(c, std::max(capacity, 0));
    if (kps && m > 0)
        GLS_CUDA(cudaMemcpyAsync(kps, s->slot[slot].kps.p, size_t(m) * sizeof(gls_keypoint), cudaMemcpyDeviceToHost, st));
    if (desc && m > 0)
        GLS_CUDA(cudaMemcpyAsync(desc, s->slot[slot].desc.p, size_t(m) * 64 * sizeof(float), cudaMemcpyDeviceToHost,
                                 st));
    GLS_CUDA(cudaStreamSynchronize(st));
    return GLS_OK;
}

gls_status gls_surf_load_features(gls_surf* s, int32_t slot, const gls_keypoint* kps, const float* desc, int32_t n,
                                  uint32_t flags, void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (slot < 0 || slot >= GLS_SURF_SLOTS) return set_error(GLS_ERR_INVALID_ARG, "slot %d out of range", slot);
    if (n < 0 || n > s->capacity)
        return set_error(GLS_ERR_INVALID_ARG, "%d features, the detector keeps at most %d", n, s->capacity);
    if (n > 0 && (!kps || !desc)) return set_error(GLS_ERR_INVALID_ARG, "NULL features");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const cudaMemcpyKind kind = (flags & GLS_HOST_IO) ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    SurfSlotState& sl = s->slot[slot];
    if (n > 0) {
        GLS_CUDA(cudaMemcpyAsync(sl.kps.p, kps, size_t(n) * sizeof(gls_keypoint), kind, st));
        GLS_CUDA(cudaMemcpyAsync(sl.desc.p, desc, size_t(n) * 64 * sizeof(float), kind, st));
    }
    // the count is written by a kernel on the stream (no host buffer has to
    // outlive the call, and the write can be recorded in a graph)
    k_store_count<<<1, 1, 0, st>>>(static_cast<int*>(sl.count.p), n);
    GLS_TRY(launch_check(s, "store_count"));
    if (flags & (GLS_SYNC | GLS_HOST_IO)) GLS_CUDA(cudaStreamSynchronize(st));
    sl.count_host = n;
    sl.valid = true;
    if (s->match_query == slot || s->match_train == slot) s->match_query = s->match_train = -1;
    return GLS_OK;
}

gls_status gls_surf_plane(gls_surf* s, int32_t which, gls_image_view* view) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (!view) return set_error(GLS_ERR_INVALID_ARG, "NULL view");
    if (which != GLS_SURF_PLANE_INTEGRAL) return set_error(GLS_ERR_INVALID_ARG, "unknown plane %d", which);
    *view = gls_image_view{s->sum.p, s->W + 1, s->H + 1, 1, GLS_F32, size_t(s->W + 1) * sizeof(float)};
    return GLS_OK;
}

gls_status gls_surf_match(gls_surf* s, int32_t query_slot, int32_t train_slot, gls_match* matches, int32_t capacity,
                          int32_t* n, void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (query_slot < 0 || query_slot >= GLS_SURF_SLOTS || train_slot < 0 || train_slot >= GLS_SURF_SLOTS)
        return set_error(GLS_ERR_INVALID_ARG, "slot out of range");
    if (!s->slot[query_slot].valid || !s->slot[train_slot].valid)
        return set_error(GLS_ERR_INVALID_ARG, "slot holds no detection");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    GLS_TRY(run_match(s, {{query_slot, train_slot}}, st));
    s->match_query = query_slot;
    s->match_train = train_slot;
    if (matches || n) {
        int c = 0;
        GLS_TRY(slot_count(s, query_slot, st, &c));
        if (n) *n = c;
        const int m = std::min(c, std::max(capacity, 0));
        if (matches && m > 0)
            GLS_CUDA(cudaMemcpyAsync(matches, s->matches_sorted.p, size_t(m) * sizeof(gls_match),
                                     cudaMemcpyDeviceToHost, st));
        GLS_CUDA(cudaStreamSynchronize(st));
    }
    return GLS_OK;
}

gls_status gls_surf_find_homography(gls_surf* s, float threshold, int32_t max_iterations, float* H, int32_t* inliers,
                                    int32_t* n_inliers, void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (!H) return set_error(GLS_ERR_INVALID_ARG, "NULL H");
    if (max_iterations < 1) return set_error(GLS_ERR_INVALID_ARG, "max_iterations must be positive");
    if (s->match_query < 0) return set_error(GLS_ERR_INVALID_ARG, "no match result (call gls_surf_match first)");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int n = 0;
    GLS_TRY(slot_count(s, s->match_query, st, &n));
    GLS_TRY(run_ransac(s, {n}, threshold, max_iterations, st));
    return ransac_result(s, H, inliers, n_inliers, st);
}

gls_status gls_find_homography(gls_surf* ctx, const float* pairs, int32_t n, float threshold, int32_t max_iterations,
                               float* H, int32_t* inliers, int32_t* n_inliers, void* stream) {
    clear_error();
    GLS_TRY(check_surf(ctx));
    if (!pairs || !H) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (max_iterations < 1) return set_error(GLS_ERR_INVALID_ARG, "max_iterations must be positive");
    if (n < 4) return set_error(GLS_ERR_DEGENERATE, "RANSAC needs at least 4 point pairs, got %d", n);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    GLS_TRY(ensure_pairs(ctx, 1, n));
    GLS_CUDA(cudaMemcpyAsync(ctx->pairs.p, pairs, size_t(n) * sizeof(float4), cudaMemcpyHostToDevice, st));
    ctx->match_query = ctx->match_train = -1;  // the pair buffer now holds host pairs
    GLS_TRY(run_ransac(ctx, {n}, threshold, max_iterations, st));
    return ransac_result(ctx, H, inliers, n_inliers, st);
}

gls_status gls_surf_register_frames(gls_surf* s, const int32_t* ref_slots, int32_t n_channels,
                                    const int32_t* frame_slots, int32_t n_frames, float threshold,
                                    int32_t max_iterations, int32_t scale_to_full, float* H, void* stream) {
    clear_error();
    GLS_TRY(check_surf(s));
    if (!ref_slots || !frame_slots || !H) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (n_channels < 1 || n_frames < 1 || n_channels * n_frames > kMaxJobs)
        return set_error(GLS_ERR_INVALID_ARG, "n_channels x n_frames must be 1..%d", kMaxJobs);
    if (max_iterations < 1) return set_error(GLS_ERR_INVALID_ARG, "max_iterations must be positive");
    auto ok = [&](int sl) { return sl >= 0 && sl < GLS_SURF_SLOTS && s->slot[sl].valid; };
    for (int c = 0; c < n_channels; c++)
        if (!ok(ref_slots[c])) return set_error(GLS_ERR_INVALID_ARG, "reference slot %d holds no detection", ref_slots[c]);
    for (int i = 0; i < n_channels * n_frames; i++)
        if (!ok(frame_slots[i])) return set_error(GLS_ERR_INVALID_ARG, "frame slot %d holds no detection", frame_slots[i]);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    std::vector<std::pair<int, int>> qt;
    std::vector<int> ns;
    for (int f = 0; f < n_frames; f++)
        for (int c = 0; c < n_channels; c++) {
            qt.push_back({ref_slots[c], frame_slots[f * n_channels + c]});
            int n = 0;
            GLS_TRY(slot_count(s, ref_slots[c], st, &n));
            ns.push_back(n);
        }
    GLS_TRY(run_match(s, qt, st));
    s->match_query = s->match_train = -1;
    GLS_TRY(run_ransac(s, ns, threshold, max_iterations, st));
    std::vector<float> Hj(qt.size() * 9);
    GLS_CUDA(cudaMemcpyAsync(Hj.data(), s->Hdev.p, Hj.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
    GLS_CUDA(cudaStreamSynchronize(st));
    for (int f = 0; f < n_frames; f++) {
        float acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int c = 0; c < n_channels; c++)  // running average, pyramidFusion.cpp:338-339
            for (int i = 0; i < 9; i++)
                acc[i] = (Hj[size_t(f * n_channels + c) * 9 + i] + acc[i] * float(c)) / float(c + 1);
        if (scale_to_full) GLS_TRY(gls_scale_homography(acc, 2.0f, acc));
        std::memcpy(H + size_t(f) * 9, acc, sizeof(acc));
    }
    return GLS_OK;
}

gls_status gls_scale_homography(const float* H, float scale, float* out) {
    (void)scale;  // Homography.hpp:30-34 ignores it
    if (!H || !out) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    const float h[9] = {H[0], H[1], H[2] * 2.0f, H[3], H[4], H[5] * 2.0f, H[6] * 0.5f, H[7] * 0.5f, H[8]};
    std::memcpy(out, h, sizeof(h));
    return GLS_OK;
}

gls_status gls_raw_channels(gls_surf* ctx, const uint16_t* raw, int32_t width, int32_t height, size_t stride_bytes,
                            int32_t bayer_pattern, float black_level, float white_level, float exposure_multiplier,
                            uint32_t channel_mask, gls_image_view* out, uint32_t flags, void* stream) {
    clear_error();
    GLS_TRY(check_surf(ctx));
    if (!raw || !out) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (bayer_pattern < 0 || bayer_pattern > 3) return set_error(GLS_ERR_INVALID_ARG, "bad Bayer pattern");
    if (width < 2 || height < 2) return set_error(GLS_ERR_INVALID_ARG, "raw image too small");
    if ((channel_mask & 0xfu) == 0 || (channel_mask & ~0xfu)) return set_error(GLS_ERR_INVALID_ARG, "bad channel mask");
    const size_t stride = stride_bytes ? stride_bytes : size_t(width) * 2;
    if (stride % 2 || stride < size_t(width) * 2) return set_error(GLS_ERR_INVALID_ARG, "bad raw stride");
    const int ow = width / 2, oh = height / 2;
    ChanArgs a{};
    static const int kHostBayer[4][4][2] = {{{1, 0}, {0, 0}, {0, 1}, {1, 1}},
                                            {{0, 1}, {0, 0}, {1, 0}, {1, 1}},
                                            {{0, 0}, {1, 0}, {1, 1}, {0, 1}},
                                            {{1, 1}, {1, 0}, {0, 0}, {0, 1}}};
    for (int c = 0; c < 4; c++) {
        a.ox[c] = kHostBayer[bayer_pattern][c][0];
        a.oy[c] = kHostBayer[bayer_pattern][c][1];
        if (!(channel_mask & (1u << c))) continue;
        const gls_image_view& v = out[c];
        if (!v.data || v.channels != 1 || v.dtype != GLS_F32 || v.width != ow || v.height != oh)
            return set_error(GLS_ERR_INVALID_ARG, "output %d must be a %dx%d single-channel GLS_F32 view", c, ow, oh);
        const size_t os = v.stride_bytes ? v.stride_bytes : size_t(ow) * 4;
        if (os % 4 || os < size_t(ow) * 4) return set_error(GLS_ERR_INVALID_ARG, "bad output stride");
        a.out[c] = reinterpret_cast<float*>(v.data);
        a.out_pitch[c] = int(os / 4);
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!(ctx->lut_black == black_level && ctx->lut_white == white_level && ctx->lut_exp == exposure_multiplier)) {
        ctx->lut_host.resize(65536);
        for (int v = 0; v < 65536; v++) {
            const float x = exposure_multiplier * (float(v) - black_level) / white_level;
            ctx->lut_host[v] = tone_curve(std::clamp(x, 0.0f, 1.0f), 3.5f);
        }
        GLS_TRY(ctx->lut.ensure(65536 * sizeof(float)));
        GLS_CUDA(cudaMemcpyAsync(ctx->lut.p, ctx->lut_host.data(), 65536 * sizeof(float), cudaMemcpyHostToDevice, st));
        ctx->lut_black = black_level;
        ctx->lut_white = white_level;
        ctx->lut_exp = exposure_multiplier;
    }
    const uint16_t* src = raw;
    size_t spx = stride / 2;
    if (flags & GLS_HOST_IO) {
        GLS_TRY(ctx->raw.ensure(size_t(width) * height * 2));
        GLS_CUDA(cudaMemcpy2DAsync(ctx->raw.p, size_t(width) * 2, raw, stride, size_t(width) * 2, height,
                                   cudaMemcpyHostToDevice, st));
        src = reinterpret_cast<const uint16_t*>(ctx->raw.p);
        spx = width;
    }
    a.raw = src;
    a.stride = spx;
    a.ow = ow;
    a.oh = oh;
    a.mask = channel_mask;
    a.lut = reinterpret_cast<const float*>(ctx->lut.p);
    k_raw_channels<<<dim3((ow + 255) / 256, oh), 256, 0, st>>>(a);
    GLS_TRY(launch_check(ctx, "k_raw_channels"));
    if (flags & (GLS_SYNC | GLS_HOST_IO)) GLS_CUDA(cudaStreamSynchronize(st));
    return GLS_OK;
}

static gls_status warp(const gls_image_view* fused, const gls_image_view* input, gls_image_view* out, const float* H,
                       int count, void* stream) {
    if (!input || !out || !H || !input->data || !out->data) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (input->channels != 4 || (input->dtype != GLS_F32 && input->dtype != GLS_F16))
        return set_error(GLS_ERR_INVALID_ARG, "input must be RGBA GLS_F32 or GLS_F16");
    if (out->channels != 4 || out->dtype != GLS_F32) return set_error(GLS_ERR_INVALID_ARG, "out must be RGBA GLS_F32");
    if (input->width < 1 || input->height < 1 || out->width < 1 || out->height < 1)
        return set_error(GLS_ERR_INVALID_ARG, "empty image");
    const size_t ies = input->dtype == GLS_F32 ? 4 : 2;
    const size_t is = input->stride_bytes ? input->stride_bytes : size_t(input->width) * 4 * ies;
    const size_t os = out->stride_bytes ? out->stride_bytes : size_t(out->width) * 16;
    if (is % (4 * ies) || os % 16 || (reinterpret_cast<uintptr_t>(input->data) % (4 * ies)) ||
        (reinterpret_cast<uintptr_t>(out->data) % 16))
        return set_error(GLS_ERR_INVALID_ARG, "pixel rows must be aligned to whole RGBA pixels");
    WarpArgs a{};
    if (count > 0) {
        if (!fused || !fused->data || fused->channels != 4 || fused->dtype != GLS_F32 || fused->width != out->width ||
            fused->height != out->height)
            return set_error(GLS_ERR_INVALID_ARG, "fused must be RGBA GLS_F32 of the output's size");
        const size_t fs = fused->stride_bytes ? fused->stride_bytes : size_t(fused->width) * 16;
        if (fs % 16 || (reinterpret_cast<uintptr_t>(fused->data) % 16))
            return set_error(GLS_ERR_INVALID_ARG, "fused rows must be 16-byte aligned");
        a.fused = reinterpret_cast<const float*>(fused->data);
        a.fused_pitch = int(fs / 4);
    }
    a.input = input->data;
    a.in_pitch = int(is / ies);
    a.iw = input->width;
    a.ih = input->height;
    a.out = reinterpret_cast<float*>(out->data);
    a.out_pitch = int(os / 4);
    a.w = out->width;
    a.h = out->height;
    for (int i = 0; i < 9; i++) a.H[i] = H[i];
    a.count = count;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid((out->width + 255) / 256, out->height);
    if (input->dtype == GLS_F32) k_register<float><<<grid, 256, 0, st>>>(a);
    else k_register<__half><<<grid, 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(GLS_ERR_CUDA, "k_register launch: %s", cudaGetErrorString(e));
    return GLS_OK;
}

gls_status gls_register_and_fuse(const gls_image_view* fused, const gls_image_view* input, gls_image_view* out,
                                 const float* H, int32_t count, void* stream) {
    clear_error();
    if (count < 1) return set_error(GLS_ERR_INVALID_ARG, "count must be >= 1");
    return warp(fused, input, out, H, count, stream);
}

gls_status gls_fuse_pyramid(gls_surf* ctx, const gls_image_view* frames, int32_t n_frames, const float* H,
                            int32_t levels, float robustness, gls_image_view* out, void* stream) {
    clear_error();
    GLS_TRY(check_surf(ctx));
    if (!frames || !out || !out->data || (n_frames > 1 && !H)) return set_error(GLS_ERR_INVALID_ARG, "NULL argument");
    if (n_frames < 1) return set_error(GLS_ERR_INVALID_ARG, "no frames");
    if (levels < 1 || levels > GLS_MAX_LEVELS) return set_error(GLS_ERR_INVALID_ARG, "levels must be 1..%d", GLS_MAX_LEVELS);
    if (!(robustness >= 0.f)) return set_error(GLS_ERR_INVALID_ARG, "robustness must be >= 0");
    const int W = frames[0].width, Hh = frames[0].height;
    if ((W >> (levels - 1)) < 1 || (Hh >> (levels - 1)) < 1) return set_error(GLS_ERR_INVALID_ARG, "too many levels");
    if (out->width != W || out->height != Hh || out->channels != 4 || (out->dtype != GLS_F32 && out->dtype != GLS_F16))
        return set_error(GLS_ERR_INVALID_ARG, "out must be a %dx%d RGBA GLS_F32 or GLS_F16 view", W, Hh);
    const size_t oes = out->dtype == GLS_F32 ? 4 : 2;
    if ((out->stride_bytes && out->stride_bytes % (4 * oes)) || (reinterpret_cast<uintptr_t>(out->data) % (4 * oes)))
        return set_error(GLS_ERR_INVALID_ARG, "out rows must be aligned to whole RGBA pixels");
    if (!ctx->fusion) ctx->fusion = fusion_scratch_new();
    return fuse_pyramid_impl(ctx->fusion, frames, n_frames, H, levels, robustness, out,
                             reinterpret_cast<cudaStream_t>(stream));
}

gls_status gls_register_image(const gls_image_view* input, gls_image_view* out, const float* H, void* stream) {
    clear_error();
    return warp(nullptr, input, out, H, 0, stream);
}

}  // extern "C"
