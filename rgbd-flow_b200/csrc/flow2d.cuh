// flow2d.cuh — 2-D optical flow on the device: Ce Liu's coarse-to-fine solver, the reference
// demo's flow type 1 (OpticalFlow::Coarse2FineFlow, src/opticalFlowMultiscale.cpp:4-146, with
// OpticalFlow::SmoothFlowSOR, src/SmoothFlowSOR.cpp:8-247).
//
// The reference's solver is numerically fragile (lexicographic SOR with omega 1.8): reordering
// its sweep changes the result by pixels on ordinary scenes.  So this solve keeps the
// reference's arithmetic exactly: FP64, every operation rounded on its own (explicit __d*_rn
// intrinsics, no fused multiply-adds), the reference's operation order, and its lexicographic
// SOR order, run as a pipeline of sweeps (k_sor_pipeline).
//
// Data: planar FP64 per level; colour pyramids 3 channels interleaved (as DImage), features 5
// channels interleaved.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>

namespace rgbdflow {
namespace f2d {

constexpr int kThreads = 256;
constexpr int kMaxRing = 16;  // sor_ring's upper limit (accepted for callers that set it; nothing depends on it)
constexpr int kMaxTaps = 64;

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ int clampi(int x, int n) { return min(max(x, 0), n - 1); }
// std::max(a, b) of the C++ library: (a < b) ? b : a (a NaN b is dropped, a NaN a is kept)
__device__ __forceinline__ double cmax(double a, double b) { return (a < b) ? b : a; }

// ImageProcessing::BilinearInterpolate, accumulating form (ImageProcessing.h:128-148)
__device__ __forceinline__ void bilinear_acc(const double* img, int W, int H, int C, double x, double y, double* out)
{
    const int xx = (int)x, yy = (int)y;
    double dx = dsub(x, (double)xx);
    if (dx > 1) dx = 1;
    if (dx < 0) dx = 0;
    double dy = dsub(y, (double)yy);
    if (dy > 1) dy = 1;
    if (dy < 0) dy = 0;
    for (int m = 0; m <= 1; m++)
        for (int n = 0; n <= 1; n++) {
            const int u = clampi(xx + m, W), v = clampi(yy + n, H);
            const size_t off = ((size_t)v * W + u) * C;
            const double s = dmul(fabs(dsub((double)(1 - m), dx)), fabs(dsub((double)(1 - n), dy)));
            for (int l = 0; l < C; l++) out[l] = dadd(out[l], dmul(img[off + l], s));
        }
}

// colour / 255 (cv2liuBGR, src/ceLiuOpticalFlow.cpp:19-37)
__global__ void k_unpack(const uint8_t* __restrict__ bgr, double* __restrict__ out, size_t n)
{
    for (size_t z = blockIdx.x * (size_t)blockDim.x + threadIdx.x; z < n; z += (size_t)gridDim.x * blockDim.x)
        out[z] = ddiv((double)bgr[z], 255.0);
}

// ImageProcessing::hfiltering / vfiltering with clamp-to-edge (ImageProcessing.h:247-269, 339-358)
__global__ void k_hfilter(const double* __restrict__ in, double* __restrict__ out, int W, int H, int C,
                          const double* __restrict__ taps, int fs)
{
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        for (int k = 0; k < C; k++) {
            double acc = 0;
            for (int l = -fs; l <= fs; l++)
                acc = dadd(acc, dmul(in[((size_t)i * W + clampi(j + l, W)) * C + k], taps[l + fs]));
            out[p * C + k] = acc;
        }
    }
}
__global__ void k_vfilter(const double* __restrict__ in, double* __restrict__ out, int W, int H, int C,
                          const double* __restrict__ taps, int fs)
{
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        for (int k = 0; k < C; k++) {
            double acc = 0;
            for (int l = -fs; l <= fs; l++)
                acc = dadd(acc, dmul(in[((size_t)clampi(i + l, H) * W + j) * C + k], taps[l + fs]));
            out[p * C + k] = acc;
        }
    }
}

// ImageProcessing::ResizeImage (ImageProcessing.h:203-242): dst (j, i) samples src at
// ((j + 1) / xr - 1, (i + 1) / yr - 1)
__global__ void k_resize(const double* __restrict__ in, int W, int H, int C, double* __restrict__ out, int DW, int DH,
                         double xr, double yr)
{
    const size_t n = (size_t)DW * DH;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / DW), j = (int)(p % DW);
        double acc[5] = {0, 0, 0, 0, 0};
        const double x = dsub(ddiv((double)(j + 1), xr), 1.0), y = dsub(ddiv((double)(i + 1), yr), 1.0);
        bilinear_acc(in, W, H, C, x, y, acc);
        for (int k = 0; k < C; k++) out[p * C + k] = acc[k];
    }
}

// Image::desaturate (Image.h:1438-1469): .114 B + .587 G + .299 R, channels in BGR order
__device__ __forceinline__ double gray_at(const double* im, size_t p)
{
    return dadd(dadd(dmul(im[p * 3], .114), dmul(im[p * 3 + 1], .587)), dmul(im[p * 3 + 2], .299));
}

// OpticalFlow::im2feature RGB_WITH_GRADIENT (OpticalFlow.cpp:189-214): gray, its 5-tap dx, dy,
// G - B, G - R
__global__ void k_features(const double* __restrict__ im, double* __restrict__ feat, int W, int H,
                           const double* __restrict__ d5)
{
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        double gx = 0, gy = 0;
        for (int l = -2; l <= 2; l++) gx = dadd(gx, dmul(gray_at(im, (size_t)i * W + clampi(j + l, W)), d5[l + 2]));
        for (int l = -2; l <= 2; l++) gy = dadd(gy, dmul(gray_at(im, (size_t)clampi(i + l, H) * W + j), d5[l + 2]));
        feat[p * 5 + 0] = gray_at(im, p);
        feat[p * 5 + 1] = gx;
        feat[p * 5 + 2] = gy;
        feat[p * 5 + 3] = dsub(im[p * 3 + 1], im[p * 3]);
        feat[p * 5 + 4] = dsub(im[p * 3 + 1], im[p * 3 + 2]);
    }
}

// x *= s (Image::Multiplywith, Image.h:1778-1782)
__global__ void k_scale(double* __restrict__ x, size_t n, double s)
{
    for (size_t z = blockIdx.x * (size_t)blockDim.x + threadIdx.x; z < n; z += (size_t)gridDim.x * blockDim.x)
        x[z] = dmul(x[z], s);
}

// warpFL, bilinear (src/opticalFlowUtils.cpp:62-67; ImageProcessing::warpImage,
// ImageProcessing.h:472-491): Im2 at (j + u, i + v), Im1 where that falls outside
__global__ void k_warp(const double* __restrict__ f1, const double* __restrict__ f2, const double* __restrict__ u,
                       const double* __restrict__ v, double* __restrict__ out, int W, int H)
{
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        const double x = dadd((double)j, u[p]), y = dadd((double)i, v[p]);
        double acc[5] = {0, 0, 0, 0, 0};
        if (x < 0 || x > W - 1 || y < 0 || y > H - 1) {
            for (int k = 0; k < 5; k++) acc[k] = f1[p * 5 + k];
        } else {
            bilinear_acc(f2, W, H, 5, x, y, acc);
        }
        for (int k = 0; k < 5; k++) out[p * 5 + k] = acc[k];
    }
}

// One level's per-iteration state.
struct LevelBufs {
    const double *f1, *f2;  // features of frames 1 and 2 (5 channels)
    double* warp;           // frame 2 features warped by the flow (5 channels)
    double *u, *v, *du, *dv, *phi;
    double *dxy, *dx2, *dy2, *dtdx, *dtdy;
    double2* coef; // the SOR's coefficients: four planes of W H pairs, each in diagonal order
                   // (written by k_rhs; read-only during the SOR)
    int W, H;
};

// 0.4 Im1 + 0.6 warp at pixel p, channel k (getDxs, src/opticalFlowUtils.cpp:33-37)
__device__ __forceinline__ double mix_at(const LevelBufs& b, size_t p, int k)
{
    return dadd(dmul(b.f1[p * 5 + k], 0.4), dmul(b.warp[p * 5 + k], 0.6));
}

// SmoothFlowSOR.cpp:52-139 for one inner iteration: the flow gradient weight phi of u + du
// (forward differences, Image::dx/dy, Image.h:955-1019), and the robust data weights psi of the
// derivatives of getDxs (5-tap dx, dy of 0.4 Im1 + 0.6 warp, dt = warp - Im1), multiplied out
// and averaged over the channels (Image::Multiply, Image::collapse).  first: the inner
// iteration's uu is u itself.
// eps: pow(0.001, 2) as the host's pow computes it (SmoothFlowSOR.cpp:30-31).
__global__ void k_phi_psi(LevelBufs b, const double* __restrict__ d5, int first, double eps)
{
    const int W = b.W, H = b.H;
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        auto uu = [&](size_t q) { return first ? b.u[q] : dadd(b.u[q], b.du[q]); };
        auto vv = [&](size_t q) { return first ? b.v[q] : dadd(b.v[q], b.dv[q]); };
        const double ux = (j < W - 1) ? dsub(uu(p + 1), uu(p)) : 0.0;
        const double uy = (i < H - 1) ? dsub(uu(p + W), uu(p)) : 0.0;
        const double vx = (j < W - 1) ? dsub(vv(p + 1), vv(p)) : 0.0;
        const double vy = (i < H - 1) ? dsub(vv(p + W), vv(p)) : 0.0;
        const double t = dadd(dadd(dadd(dmul(ux, ux), dmul(uy, uy)), dmul(vx, vx)), dmul(vy, vy));
        b.phi[p] = ddiv(0.5, __dsqrt_rn(dadd(t, eps)));
        const double du = first ? 0.0 : b.du[p], dv = first ? 0.0 : b.dv[p];
        double sxy = 0, sx2 = 0, sy2 = 0, stx = 0, sty = 0;
        for (int k = 0; k < 5; k++) {
            double ix = 0, iy = 0;
            for (int l = -2; l <= 2; l++) ix = dadd(ix, dmul(mix_at(b, (size_t)i * W + clampi(j + l, W), k), d5[l + 2]));
            for (int l = -2; l <= 2; l++) iy = dadd(iy, dmul(mix_at(b, (size_t)clampi(i + l, H) * W + j, k), d5[l + 2]));
            const double it = dsub(b.warp[p * 5 + k], b.f1[p * 5 + k]);
            double r = dadd(dadd(it, dmul(ix, du)), dmul(iy, dv));
            r = dmul(r, r);
            const double psi = ddiv(1.0, dmul(2.0, __dsqrt_rn(dadd(r, eps))));
            sxy = dadd(sxy, dmul(dmul(psi, ix), iy));
            sx2 = dadd(sx2, dmul(dmul(psi, ix), ix));
            sy2 = dadd(sy2, dmul(dmul(psi, iy), iy));
            stx = dadd(stx, dmul(dmul(psi, ix), it));
            sty = dadd(sty, dmul(dmul(psi, iy), it));
        }
        b.dxy[p] = ddiv(sxy, 5.0);
        b.dx2[p] = ddiv(sx2, 5.0);
        b.dy2[p] = ddiv(sy2, 5.0);
        b.dtdx[p] = ddiv(stx, 5.0);
        b.dtdy[p] = ddiv(sty, 5.0);
    }
}

// Laplacian with normalising weights (src/opticalFlowUtils.cpp:252-313) of x at pixel (i, j),
// weighted by the 1-channel phi read as a 2-channel image, as SmoothFlowSOR.cpp:144 calls it:
// channel k of (i, j) is element i * W + j + k (Image::operator(), Image.h:76).
__device__ __forceinline__ double laplacian_phi(const double* x, const double* phi, int W, int H, int i, int j)
{
    const size_t o = (size_t)i * W + j;
    double out = 0;
    if (j < W - 1) out = dsub(out, dmul(dsub(x[o + 1], x[o]), phi[o]));
    if (j > 0) out = dadd(out, dmul(dsub(x[o], x[o - 1]), phi[o - 1]));
    if (i < H - 1) out = dsub(out, dmul(dsub(x[o + W], x[o]), phi[o + 1]));
    if (i > 0) out = dadd(out, dmul(dsub(x[o], x[o - W]), phi[o - W + 1]));
    double norm = 0;
    int count = 0;
    if (j < W - 1) { norm = dadd(norm, phi[o]); count++; }
    if (j > 0) { norm = dadd(norm, phi[o - 1]); count++; }
    if (i < H - 1) { norm = dadd(norm, phi[o + 1]); count++; }
    if (i > 0) { norm = dadd(norm, phi[o - W + 1]); count++; }
    if (fabs(norm) < 1e-5) return 0;
    return ddiv(out, ddiv(norm, (double)count));
}

// Diagonal order of a W x H image: diagonal d = i + j after diagonal, each by row.  The element of pixel
// (i, d - i) is diag_base(d) + i.
__host__ __device__ inline int diag_start(int d, int W, int H)
{
    const int a = W < H ? W : H, b = W < H ? H : W;
    if (d <= 0) return 0;
    if (d <= a) return d * (d + 1) / 2;
    if (d <= b) return a * (a + 1) / 2 + (d - a) * a;
    const int r = W + H - 1 - d;
    return r <= 0 ? W * H : W * H - r * (r + 1) / 2;
}
__host__ __device__ inline int diag_base(int d, int W, int H)
{
    return diag_start(d, W, H) - (d - W + 1 > 0 ? d - W + 1 : 0);
}

// The right-hand sides (SmoothFlowSOR.cpp:144-151): -Itx - alpha * Lap(u), -Ity - alpha * Lap(v), and what an
// SOR update (SmoothFlowSOR.cpp:166-215) reads of a pixel that no sweep changes: omega over the two
// denominators (the reference divides anew at every update; same operands, same quotient) and the
// neighbours' weights (0 where there is no neighbour).
constexpr double kOmega = 1.8;
__global__ void k_rhs(LevelBufs b, double alpha)
{
    const int W = b.W, H = b.H;
    const size_t n = (size_t)W * H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / W), j = (int)(p % W);
        const double tx = dsub(-b.dtdx[p], dmul(alpha, laplacian_phi(b.u, b.phi, W, H, i, j)));
        const double ty = dsub(-b.dtdy[p], dmul(alpha, laplacian_phi(b.v, b.phi, W, H, i, j)));
        const double phi = b.phi[p], phiL = j > 0 ? b.phi[p - 1] : 0.0, phiU = i > 0 ? b.phi[p - W] : 0.0;
        double ws = 0;
        if (j > 0) ws = dadd(ws, phiL);
        if (j < W - 1) ws = dadd(ws, phi);
        if (i > 0) ws = dadd(ws, phiU);
        if (i < H - 1) ws = dadd(ws, phi);
        ws = dmul(ws, alpha);
        double2* c = b.coef + diag_base(i + j, W, H) + i;
        c[0] = make_double2(b.dxy[p], ddiv(kOmega, dadd(b.dx2[p], ws)));
        c[n] = make_double2(ddiv(kOmega, dadd(b.dy2[p], ws)), tx);
        c[2 * n] = make_double2(ty, phi);
        c[3 * n] = make_double2(phiU, phiL);
    }
}

// ------------------------------------------------------------------------------------------
// The SOR iterations of one inner iteration (SmoothFlowSOR.cpp:156-226): lexicographic sweeps with omega 1.8,
// up to the first whose largest change is below 1e-5.  Pixel (i, j) of sweep s reads (i, j - 1) and
// (i - 1, j) of its own sweep, and (i, j + 1), (i + 1, j) and itself of sweep s - 1.
//
// A task is G sweeps of a band; row l of the band is, in its sweep s, image row 32 B + l - s: rows move up by
// one from sweep to sweep, so that all a row reads of sweep s - 1 lies in the band's rows l - 1 and l, and
// data flows between bands in one direction.  A warp takes one sweep, a lane one of the band's 32 rows, each
// lane one column behind the lane above: at step t lane l is at column t - l.  Then
//   * the left neighbour is the lane's own last result, the upper one the lane above's (a shuffle),
//   * the lower old value is what the warp of the sweep before put into its queue for this row, the right
//     old one what it put there for the row above (a shuffle), the pixel's own old value the right one of
//     the step before.
// So an update reads one value of the sweep before and its coefficients; sweeps follow each other two steps
// apart, a block barrier a step.  Values cross between tasks through L2: the band's last row, of each sweep,
// to the band below, and the last sweep's image to the next G sweeps.  Those areas are filled with a
// bit pattern that no operation produces (all ones) before the launch; two feeding warps poll the
// values themselves.  Tasks are numbered so that a task reads only tasks before it; CTAs take them in order
// (cooperative launch, every wait bounded).
//
// The largest change of each sweep is combined over the bands; the first sweep below 1e-5 is known once its
// last band is done, and tasks of later sweeps stop.  When it is not its group's last sweep, a second
// launch (finish) runs its group again with fewer sweeps: no result of a sweep after it is used.
//
// What bounds it: the step.  It is a chain of 15 dependent FP64 operations between two barriers, and a sweep
// starts three steps after the one before it (two for the data, one for the rows' shift), so an inner
// iteration of 400 sweeps is 1200 steps and the level's width and height.  Groups of 8 sweeps: 16 keep the FP64
// pipe (2 cycles a warp instruction) longer in a step than its chain lasts, fewer have more hand-overs
// through L2 and more tasks than SMs.  Measured, one solve, device time: 320x240 85.8 ms (16), 73.1 (12), 65.8 (8),
// 67.4 (6), 67.8 (4); 160x120 46.6, 39.4, 34.9, 34.2, 34.0.  Diagonal after diagonal over a cluster of 16 CTAs, a
// cluster barrier a step and every value through L2, it was 637 ms at 320x240.
constexpr int kPipeG = 8, kPipeThreads = 32 * (kPipeG + 2), kPipeAhead = 4;
constexpr int kPipePolls = 1 << 20;  // of a value, before a wait gives up

struct PipeArgs {
    int W, H, NB;                 // level, bands
    int s0, n, G;                 // this launch's sweeps: the first, how many, in groups of G
    double alpha;
    const double2* coef;          // four planes of W H
    double2* img;                 // images in diagonal order: slot 0 the input, slot g + 1 group g's, the last the finish's
    double2* bnd;                 // last rows: [group, then the finish][band][sweep][column]
    ulonglong2* sweep;            // of each of the launch's sweeps: largest change (bits), bands done
    int* conv;                    // first sweep below the threshold (0x7f7f7f7f: none yet; -1: a wait gave up)
    int zero_in;                  // the input is 0 (slot 0 is not read)
    int finish;
    int polls;
    int* status;                  // 1: a bounded wait gave up
};

__device__ __forceinline__ void pipe_store(double2* p, double2 v)
{
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p),
                 "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)) : "memory");
}
// Loads where `want` is set, 0 elsewhere (no branch: the loads of several steps are in flight together).
__device__ __forceinline__ double2 pipe_load(const double2* p, bool want)
{
    unsigned long long lo, hi;
    asm volatile("{\n .reg .pred w;\n .reg .b128 q;\n setp.ne.u32 w, %3, 0;\n mov.b128 q, {%4, %4};\n"
                 " @w ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(lo), "=l"(hi) : "l"(p), "r"((unsigned)want), "l"(0ull) : "memory");
    return make_double2(__longlong_as_double(lo), __longlong_as_double(hi));
}
__device__ __forceinline__ bool pipe_ready(double2 v) { return __double_as_longlong(v.x) != -1LL; }
// Brings a line of the coefficients into L1.
__device__ __forceinline__ void pipe_touch(const double2* p)
{
    asm volatile("{\n .reg .f64 a, b;\n ld.global.ca.v2.f64 {a, b}, [%0];\n}\n" ::"l"(p));
}

__global__ void __launch_bounds__(kPipeThreads, 1) k_sor_pipeline(PipeArgs a)
{
    __shared__ double2 queue[kPipeG + 1][4][32];  // [sweep + 1 (0: the group's input)][step & 3][row]
    __shared__ double2 edge[kPipeG + 1][4];       // the band above's last row: [sweep + 1][column & 3]
    __shared__ int s_conv;
    const int W = a.W, H = a.H, N = W * H, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int ng = (a.n + a.G - 1) / a.G;
    int t0 = 0, t1 = ng * a.NB, gs_finish = 0;
    if (tid == 0) s_conv = *(volatile int*)a.conv;
    __syncthreads();
    const int conv0 = s_conv;
    if (conv0 < a.s0) return;
    if (a.finish) {
        if (conv0 >= a.s0 + a.n) return;
        const int g = (conv0 - a.s0) / a.G;
        gs_finish = (conv0 - a.s0) % a.G + 1;
        if (gs_finish == min(a.G, a.n - g * a.G)) return;  // the group's own image is the result
        t0 = g * a.NB;
        t1 = t0 + a.NB;
    }
    for (int task = t0 + blockIdx.x; task < t1; task += gridDim.x) {
        const int g = task / a.NB, B = task % a.NB, slot = a.finish ? ng : g;
        const int gs = a.finish ? gs_finish : min(a.G, a.n - g * a.G);
        const double2* const in = a.img + (size_t)g * N;
        double2* const out = a.img + (size_t)(slot + 1) * N;
        double2* const bout = a.bnd + ((size_t)slot * a.NB + B) * a.G * W;
        const double2* const bin = bout - (size_t)a.G * W;  // the band above's (not read by band 0)
        const bool zero = a.zero_in && g == 0;
        const int last = W + 30 + 2 * (gs - 1);             // the last step
        bool stop = false, gave_up = false;
        __syncthreads();  // every warp has left the last task's queues
        if (w < kPipeG) {
            // ---- sweep w of the group
            const int row = 32 * B + lane - w;
            const bool rowok = w < gs && row >= 0 && row < H;
            double2 left = make_double2(0, 0), self = make_double2(0, 0);
            double2 c[2][4] = {};
            double mx = 0;
            // the diagonal of the coefficients that are read next: at first that of tau = 0
            int d = 32 * B - w, base = diag_base(d, W, H);
            auto load_coef = [&](double2* q, int j) {
                const bool ok = rowok && j >= 0 && j < W;
                const double2* p = a.coef + (ok ? base + row : 0);
#pragma unroll
                for (int z = 0; z < 4; z++) q[z] = ok ? __ldg(p + (size_t)z * N) : make_double2(0, 0);
                // to the next diagonal: past this one's elements, its first row one lower from column W - 1 on
                if (d >= 0 && d < W + H - 1) base += min(H - 1, d) - max(0, d - W + 1) + 1 - (d + 1 - W + 1 > 0 ? 1 : 0);
                d++;
            };
            if (__syncthreads_or(0)) stop = true;  // the feeding warps' first values are in place
            for (int t = -1; !stop && t <= last; t += 2) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int tt = t + h, tau = tt - 2 * w, j = tau - lane;
                    if (stop || tt > last) break;
                    if (w < gs && tau >= -1 && tau <= W + 30) {
                        double2 cc[4];
#pragma unroll
                        for (int z = 0; z < 4; z++) cc[z] = c[h][z];
                        load_coef(c[h ^ 1], j + 1);
                        const bool ok = rowok && j >= 0 && j < W;
                        double2 lo = make_double2(0, 0);
                        if (tau >= 0) lo = queue[w][tau & 3][lane];
                        double2 right, up;
                        right.x = __shfl_up_sync(0xffffffffu, lo.x, 1);
                        right.y = __shfl_up_sync(0xffffffffu, lo.y, 1);
                        up.x = __shfl_up_sync(0xffffffffu, left.x, 1);
                        up.y = __shfl_up_sync(0xffffffffu, left.y, 1);
                        if (lane == 0) {
                            right = edge[w][(tau + 1) & 3];
                            up = tau >= 0 ? edge[w + 1][tau & 3] : make_double2(0, 0);
                        }
                        const double dxy = cc[0].x, rU = cc[0].y, rV = cc[1].x, tx = cc[1].y, ty = cc[2].x, phi = cc[2].y;
                        const double wL = cc[3].y, wU = cc[3].x, wR = j < W - 1 ? phi : 0.0, wD = row < H - 1 ? phi : 0.0;
                        double sU = dadd(0.0, dmul(wL, left.x)), sV = dadd(0.0, dmul(wL, left.y));
                        sU = dadd(sU, dmul(wR, right.x)); sV = dadd(sV, dmul(wR, right.y));
                        sU = dadd(sU, dmul(wU, up.x)); sV = dadd(sV, dmul(wU, up.y));
                        sU = dadd(sU, dmul(wD, lo.x)); sV = dadd(sV, dmul(wD, lo.y));
                        sU = dadd(dmul(sU, -a.alpha), dmul(dxy, self.y));
                        sV = dmul(sV, -a.alpha);
                        const double nU = dadd(dmul(1 - kOmega, self.x), dmul(rU, dsub(tx, sU)));
                        sV = dadd(sV, dmul(dxy, nU));
                        const double nV = dadd(dmul(1 - kOmega, self.y), dmul(rV, dsub(ty, sV)));
                        const double m = cmax(fabs(dsub(nU, self.x)), fabs(dsub(nV, self.y)));
                        if (ok && m > mx) mx = m;  // a NaN is skipped, as std::max skips it
                        left = ok ? make_double2(nU, nV) : make_double2(0, 0);
                        self = right;
                        if (tau >= 0) queue[w + 1][tau & 3][lane] = left;
                        if (ok && lane == 31) pipe_store(bout + (size_t)w * W + j, left);
                        if (ok && w == gs - 1) pipe_store(out + diag_base(row + j, W, H) + row, left);
                    }
                    if (__syncthreads_or(0)) stop = true;
                }
            }
            if (!stop && w < gs && !a.finish) {
                // bits of a double >= 0 order as the value
                unsigned long long bits = (unsigned long long)__double_as_longlong(mx);
                for (int o = 16; o; o >>= 1) bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, o));
                if (lane == 0) {
                    const int s = g * a.G + w;
                    ulonglong2* const sw = a.sweep + s;
                    if (bits) atomicMax(&sw->x, bits);
                    __threadfence();
                    if (atomicAdd(&sw->y, 1ull) == (unsigned long long)(a.NB - 1)) {
                        __threadfence();
                        if (__longlong_as_double((long long)__ldcg(&sw->x)) < 1e-5) atomicMin(a.conv, a.s0 + s);
                    }
                }
            }
        } else {
            // ---- the feeding warps.  Warp kPipeG: the group's input for the band's rows (image rows 32 B + lane + 1),
            // column t + 1 - lane.  The next: lanes 0..G the band above's last row of sweep lane - 1 (lane 0:
            // the input's row 32 B), column t + 1 - 2 (lane - 1)
            const bool image = w == kPipeG;
            const int q = lane - 1, row = image ? 32 * B + lane + 1 : 32 * B - 1 - q;
            const bool from_image = image || lane == 0;
            const bool rowok = row >= 0 && row < H && (from_image ? !zero : (B > 0 && lane <= gs));
            auto col = [&](int t) { return image ? t + 1 - lane : t + 1 - 2 * q; };
            auto wants = [&](int t) { const int c = col(t); return rowok && c >= 0 && c < W; };
            auto at = [&](int t) {
                const int c = col(t);
                if (!wants(t)) return (const double2*)a.coef;
                return from_image ? in + diag_base(row + c, W, H) + row : bin + (size_t)q * W + c;
            };
            auto poll = [&](int t, double2 v) {
                for (int k = 0; !pipe_ready(v); k++) {
                    if (k >= a.polls) { gave_up = true; break; }
                    if ((k & 15) == 15 && *(volatile int*)a.conv < (a.finish ? 0 : a.s0 + g * a.G)) { stop = true; break; }
                    v = pipe_load(at(t), true);
                }
                return v;
            };
            // the coefficients that the sweeps read eight steps later into L1: the first sweep's rows, and the
            // first row of the others'
            auto touch = [&](int t) {
                const int s = image ? 0 : lane - kPipeG, i = image ? 32 * B + lane : 32 * B - s, j = t + 8 - 2 * s - (image ? lane : 0);
                if ((image || (s > 0 && s < gs)) && i >= 0 && i < H && j >= 0 && j < W) {
                    const double2* p = a.coef + diag_base(i + j, W, H) + i;
#pragma unroll
                    for (int z = 0; z < 4; z++) pipe_touch(p + (size_t)z * N);
                }
            };
            auto put = [&](int t, double2 v) {
                if (image) queue[0][(t + 1) & 3][lane] = v;
                else if (lane <= kPipeG) edge[lane][col(t) & 3] = v;
            };
            for (int t = -9; t < -1; t++) touch(t);
            // the input's row 32 B is a sweep ahead of the others: its first two columns now
            if (!image && lane == 0)
                for (int t = -3; t < -1; t++) put(t, wants(t) ? poll(t, pipe_load(at(t), true)) : make_double2(0, 0));
            double2 v[kPipeAhead];
#pragma unroll
            for (int k = 0; k < kPipeAhead; k++) v[k] = pipe_load(at(k - 1), wants(k - 1));
            if (__syncthreads_or(stop || gave_up)) stop = true;
            for (int t = -1; !stop && t <= last; t += kPipeAhead) {
#pragma unroll
                for (int k = 0; k < kPipeAhead; k++) {
                    if (stop || t + k > last) break;
                    double2 x = v[k];
                    if (wants(t + k)) x = poll(t + k, x);
                    __syncwarp();
                    put(t + k, x);
                    v[k] = pipe_load(at(t + k + kPipeAhead), wants(t + k + kPipeAhead));
                    touch(t + k);
                    if (__syncthreads_or(stop || gave_up)) stop = true;
                }
            }
        }
        if (gave_up) {
            atomicMin(a.conv, -1);  // every other wait stops at this too
            *a.status = 1;
        }
    }
}

// The increment the sweeps end with, into (du, dv); fin: this launch group holds the last sweep.
__global__ void k_sor_result(LevelBufs b, PipeArgs a, int fin)
{
    const int conv = *a.conv;
    if (conv < a.s0 || (conv >= a.s0 + a.n && !fin)) return;
    const int last = min(conv, a.s0 + a.n - 1), g = (last - a.s0) / a.G, ng = (a.n + a.G - 1) / a.G;
    const bool whole = (last - a.s0) % a.G + 1 == min(a.G, a.n - g * a.G);
    const size_t n = (size_t)b.W * b.H;
    const double2* img = a.img + (size_t)(whole ? g + 1 : ng + 1) * n;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(p / b.W), j = (int)(p % b.W);
        const double2 x = img[diag_base(i + j, b.W, b.H) + i];
        b.du[p] = x.x;
        b.dv[p] = x.y;
    }
}

// Work space of a level's pipeline: how many groups of how many sweeps a launch takes within `avail` bytes.
struct PipePlan {
    int G, groups, NB;
    size_t img, bnd;  // bytes of an image, of a group's last rows
};
static inline PipePlan pipe_plan(int W, int H, int nSOR, size_t avail)
{
    PipePlan p{};
    for (int G = kPipeG; G >= 1; G /= 2) {
        p.G = G;
        p.NB = (H + G - 1 + 31) / 32;
        p.img = (size_t)W * H * sizeof(double2);
        p.bnd = (size_t)p.NB * G * W * sizeof(double2);
        const size_t fixed = 2 * p.img + p.bnd, per = p.img + p.bnd + G * sizeof(ulonglong2);
        if (avail < fixed + per) continue;
        p.groups = (int)std::min<size_t>((size_t)((nSOR - 1) / G + 1), (avail - fixed) / per);
        break;
    }
    return p;
}

// u += du, v += dv (Image::Add, SmoothFlowSOR.cpp:227-228)
__global__ void k_update(LevelBufs b)
{
    const size_t n = (size_t)b.W * b.H;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        b.u[p] = dadd(b.u[p], b.du[p]);
        b.v[p] = dadd(b.v[p], b.dv[p]);
    }
}

}  // namespace f2d
}  // namespace rgbdflow
