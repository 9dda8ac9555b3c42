// Input preparation on the device: the views of one group transformed into the
// deconvolution bounding box and fused, with the fusion and deconvolution blending weights
// (ProcessInputImages.fuseGroups, deconvolution/util/ProcessInputImages.java:279-399).
//
// Per output voxel p of the bounding box (world coordinate s = p + bb_min) and view v:
//   t = model_v^-1 s                                  (double, AffineTransform3D.applyInverse)
//   image  I_v = max(1, linear interpolation of the view at t) when t lies strictly inside
//                the view (min < t < max on every axis), else 0
//                (TransformView.transformView with minValueImg 1 / outsideValueImg 0,
//                 TransformedInputRandomAccess.get, AbstractTransformedImgRandomAccess)
//   weights wf_v, wd_v = the cosine blending of the view's interval at t (as float) with the
//                fusion / deconvolution border and range, or 1 without blending
//                (TransformWeight.transformBlending, TransformedRasteredRandomAccess.applyInverse,
//                 BlendingRealRandomAccess.computeWeight)
//   fused image = sum(I_v wf_v) / sum(wf_v) over wf_v != 0, 0 when the sum is 0
//                (FusedRandomAccess.get, Fusion.AVG)
//   deconvolution weight = sum(wd_v) (CombineWeightsSumRandomAccess.get)
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/mvr_gb300.h"
#include "affine.cuh"

namespace mvr {
namespace {

constexpr int kFuseMaxViews = 16;
constexpr int kFuseRows = 8;        // rows of one plane a CTA takes at a time
constexpr int kFuseThreads = 256;
constexpr int kFuseLong = 1 << 24;  // a row's x is a float up to here

// ---- pairs of floats (hi + lo, about 48 bits) ------------------------------------------------
// The GPU's double rate is a small fraction of its float rate: one fused voxel in double (affine
// map, eight corner weights, table products) took 13.1 ms for 3 views into a 256^3 box.  The sums
// and products that decide a rounding or a branch run on pairs of floats instead; the products'
// and sums' rounding errors come from fused multiply-adds and two-sums (Dekker, Knuth).
struct FPair {
    float h, l;
};
__host__ __device__ __forceinline__ FPair fp_from(double v)
{
    FPair p;
    p.h = (float)v;
    p.l = (float)(v - (double)p.h);
    return p;
}
__device__ __forceinline__ FPair fp_quick(float a, float b)  // |a| >= |b|
{
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FPair fp_sum(float a, float b)
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FPair fp_add(FPair a, FPair b)
{
    const FPair s = fp_sum(a.h, b.h);
    return fp_quick(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ FPair fp_mul(FPair a, float b)
{
    const float p = __fmul_rn(a.h, b);
    return fp_quick(p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p)));
}
__device__ __forceinline__ FPair fp_prod(float a, float b)
{
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

// The blending look-up table of BlendingRealRandomAccess: d runs from 0 in steps of 0.001 (accumulated
// in double, as there), entry (int)(d * 1000 + 0.5) = (cos((1 - d) pi) + 1) / 2.  Every call puts the
// same values into the module's table (no allocation; calls on other streams may read it meanwhile).
constexpr int kLut = 1001;
__device__ FPair d_lut[kLut];
const std::vector<FPair> &blending_lut()
{
    static const std::vector<FPair> lut = [] {
        std::vector<FPair> t(kLut, FPair{0.0f, 0.0f});
        for (double d = 0; d <= 1.0001; d = d + 0.001) t[(int)(d * 1000.0 + 0.5)] = fp_from((std::cos((1 - d) * M_PI) + 1) / 2);
        return t;
    }();
    return lut;
}

struct FuseView {
    const float *img;
    int dims[3];
    double inv[12];  // world -> view pixel, row-packed 3 x 4
    FPair step[3];   // inv[0], inv[4], inv[8]: t per voxel of x
    float fb[3], fr[3], db[3], dr[3];
    float fri[3], dri[3];    // 1 / range
    float top[3], half[3];   // dims - 1, and half of it
    int fblend, dblend;
    int adjust;        // intensity adjustment v -> v m00 + m01 (rounded once to float)
    FPair m00, m01;
    double m[2];       // the same in double
};

struct FuseViews {
    FuseView v[kFuseMaxViews];
    int n;
};

// One axis of BlendingRealRandomAccess.computeWeight on an interval [0, top] at a float location l
// (float arithmetic as in the reference): the distance to the border zone, and the weight's factor
// where it is inside the range.  inv: 1 / range rounded to float; the quotient is that product
// with one residual correction (Markstein), the table entry index (int)(rel 1000 + 0.5) comes from
// the exact product rel 1000, and w lut[i] is rounded once.
__device__ __forceinline__ float blend_distance(float l, float l2, float border)  // l2 = top - l
{
    return fminf(__fsub_rn(l, border), __fsub_rn(l2, border));
}
__device__ __forceinline__ float blend_factor(float w, float dist, float range, float inv)
{
    if (!(dist < range)) return w;  // exactly the quotients that round to 1 or more
    const float q = __fmul_rn(dist, inv);
    const float rel = __fmaf_rn(__fmaf_rn(-q, range, dist), inv, q);
    const FPair p = fp_prod(rel, 1000.0f);
    float k = floorf(__fadd_rn(p.h, 0.5f));
    const float r = __fadd_rn(__fsub_rn(p.h, k), p.l);  // rel 1000 - k: p.h - k is exact
    k += r >= 0.5f ? 1.0f : (r < -0.5f ? -1.0f : 0.0f);
    const FPair c = d_lut[(int)k];
    const float ph = __fmul_rn(c.h, w);
    return __fadd_rn(ph, __fmaf_rn(c.l, w, __fmaf_rn(c.h, w, -ph)));
}

// Linear interpolation at floor(t) + f in [0, 1]^3 (all eight neighbours exist: t lies strictly
// inside) along x, y, z, with both weights u = 1 - f and f rounded from the pair that t is: a difference
// form (b - a) f + a keeps f's distance to 1 only to 2^-25, which a bright neighbour multiplies.  With `adjust` every neighbour goes
// through the intensity adjustment first (IntensityAdjuster.apply,
// fusion/intensityadjust/IntensityAdjuster.java: v m00 + m01, stored as float).
__device__ __forceinline__ float fuse_value(const FuseView &v, float x)
{
    if (!v.adjust) return x;
    const FPair q = fp_add(fp_mul(v.m00, x), v.m01);
    return __fadd_rn(q.h, q.l);
}
__device__ __forceinline__ float lerp(float a, float b, float u, float f) { return __fmaf_rn(f, b, __fmul_rn(u, a)); }
__device__ __forceinline__ float trilinear(const FuseView &v, const int *i, const float *u, const float *f)
{
    const long long sy = v.dims[0], sz = (long long)v.dims[0] * v.dims[1];
    const float *p = v.img + ((long long)i[2] * v.dims[1] + i[1]) * sy + i[0];
    float c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = __ldg(p + (k & 1) + (k & 2 ? sy : 0) + (k & 4 ? sz : 0));
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = fuse_value(v, c[k]);
    const float y0 = lerp(lerp(c[0], c[1], u[0], f[0]), lerp(c[2], c[3], u[0], f[0]), u[1], f[1]);
    const float y1 = lerp(lerp(c[4], c[5], u[0], f[0]), lerp(c[6], c[7], u[0], f[0]), u[1], f[1]);
    return lerp(y0, y1, u[2], f[2]);
}

// hi + lo += x, the rounding errors of the high part gathered in the low one
__device__ __forceinline__ void fp_gather(FPair &s, float x)
{
    const FPair t = fp_sum(s.h, x);
    s.h = t.h;
    s.l = __fadd_rn(s.l, t.l);
}

// One voxel with positions, interpolation and sums in double: for the voxels where a sample or a sum left
// the range of a float (samples that are infinite or not a number among them: the residuals of the
// pairs would turn an infinity into NaN).  In a kernel of its own behind k_fuse_group, which marks them:
// 14 us of 551 (3 views, 256^3); as a call in that kernel 16 registers and 19 us.
__device__ __forceinline__ void fuse_voxel(const FuseViews &fv, double s0, double s1, double s2, float &image, float &weight)
{
    const double s[3] = {s0, s1, s2};
    double sumI = 0.0, sumW = 0.0, sumD = 0.0;
    for (int k = 0; k < fv.n; ++k) {
        const FuseView &v = fv.v[k];
        double t[3], w[3];
        apply_affine(v.inv, s, t);
        long long at = 0;
        bool in = true;
        float dw = INFINITY, dd = INFINITY, wf = 1.0f, wd = 1.0f;
        for (int d = 2; d >= 0; --d) {
            const float tf = (float)t[d], l2 = __fsub_rn(v.top[d], tf);
            if (v.fblend) dw = fminf(dw, blend_distance(tf, l2, v.fb[d]));
            if (v.dblend) dd = fminf(dd, blend_distance(tf, l2, v.db[d]));
            const double fl = floor(t[d]);
            w[d] = __dsub_rn(t[d], fl);
            in = in && t[d] > 0.0 && t[d] < v.dims[d] - 1;
            at = at * v.dims[d] + (in ? (long long)fl : 0);
        }
        if (!(dw > 0.0f)) wf = 0.0f;
        if (!(dd > 0.0f)) wd = 0.0f;
        for (int d = 0; d < 3; ++d) {
            const float tf = (float)t[d], l2 = __fsub_rn(v.top[d], tf);
            if (wf != 0.0f && v.fblend) wf = blend_factor(wf, blend_distance(tf, l2, v.fb[d]), v.fr[d], v.fri[d]);
            if (wd != 0.0f && v.dblend) wd = blend_factor(wd, blend_distance(tf, l2, v.db[d]), v.dr[d], v.dri[d]);
        }
        sumD += (double)wd;
        if (wf == 0.0f) continue;
        float val = 0.0f;  // outsideValueImg
        if (in) {
            const float *p = v.img + at;
            const long long sy = v.dims[0], sz = (long long)v.dims[0] * v.dims[1];
            val = fmaxf(1.0f, nlinear3(w, [&](int dx, int dy, int dz) {  // minValueImg
                const float x = __ldg(p + dz * sz + dy * sy + dx);
                return v.adjust ? __double2float_rn(__dadd_rn(__dmul_rn((double)x, v.m[0]), v.m[1])) : x;
            }));
        }
        sumI += (double)val * (double)wf;
        sumW += (double)wf;
    }
    image = sumW > 0.0 ? (float)(sumI / sumW) : 0.0f;
    weight = (float)sumD;
}
// The last call that left voxels to k_fuse_wide, by its number (calls run on any stream).
constexpr int kWideCalls = 1024;
__device__ unsigned long long d_wide[kWideCalls];

// A CTA takes kFuseRows rows of the box: the part of t that is constant along a row is formed in
// double, once per row, view and axis (apply_affine at the row's first voxel), and t = base + x
// step on pairs of floats per voxel.  Bound by instruction issue (82 % of the issue slots): 3 views
// with blending into a 256^3 box 0.55 ms, 13.1 ms in double; 2 or 4 voxels of a thread at a time
// (a view's constants fetched once for them) 0.58 and 0.98 ms: the branches of the border zones
// keep them from overlapping.  Six CTAs per SM: 554 us, five 571.
__global__ void __launch_bounds__(kFuseThreads, 6)
    k_fuse_group(const __grid_constant__ FuseViews fv, long long bx, long long by, long long bz, int nx, int ny, int nz,
                 float *__restrict__ out_img, float *__restrict__ out_w, unsigned long long call)
{
    __shared__ FPair base[kFuseRows][kFuseMaxViews][3];
    const int per = nx > kFuseLong ? 1 : kFuseRows;
    const int y0 = blockIdx.x * per, z = blockIdx.y;
    const int rows = min(per, ny - y0);
    for (int i = threadIdx.x; i < rows * fv.n; i += kFuseThreads) {
        const int k = i / rows, r = i - k * rows;
        const double s[3] = {(double)bx, (double)(y0 + r + by), (double)(z + bz)};
        double t[3];
        apply_affine(fv.v[k].inv, s, t);
        for (int d = 0; d < 3; ++d) base[r][k][d] = fp_from(t[d]);
    }
    __syncthreads();
    const unsigned total = (unsigned)rows * nx;
    const long long o0 = ((long long)z * ny + y0) * nx;
    for (unsigned i = threadIdx.x; i < total; i += kFuseThreads) {
        const int row = i / nx, x = i - row * nx;
        const float xf = (float)x;
        FPair sumI = {0.0f, 0.0f}, sumW = {0.0f, 0.0f}, sumD = {0.0f, 0.0f};
        bool wide = x >= kFuseLong;  // or a sample is not finite
        for (int k = 0; k < fv.n; ++k) {
            const FuseView &v = fv.v[k];
            float f[3], u[3], dw[3], dd[3];
            int c[3];
            bool in = true;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const FPair b = base[row][k][d];
                const FPair p = fp_prod(v.step[d].h, xf), sm = fp_sum(p.h, b.h);
                FPair t = fp_quick(sm.h, __fadd_rn(sm.l, __fadd_rn(b.l, __fmaf_rn(v.step[d].l, xf, p.l))));
                // next to a face of the view (a whole plane of samples, when the views are a quarter turn
                // apart) the rounding of the double evaluation decides inside or outside: take that one
                if (fabsf(__fsub_rn(fabsf(__fsub_rn(t.h, v.half[d])), v.half[d])) < 1e-2f) {
                    const double s[3] = {(double)(x + bx), (double)(y0 + row + by), (double)(z + bz)};
                    t = fp_from(apply_affine_row(v.inv + 4 * d, s));
                }
                float fl = floorf(t.h), r = __fsub_rn(t.h, fl);
                if (r < -t.l) {  // t just below an integer
                    fl -= 1.0f;
                    r = 1.0f;
                }
                f[d] = __fadd_rn(r, t.l);
                u[d] = __fsub_rn(__fsub_rn(1.0f, r), t.l);
                c[d] = (int)fl;
                in = in && t.h > 0.0f && fl < v.top[d];
                const float l2 = __fsub_rn(v.top[d], t.h);
                dw[d] = v.fblend ? blend_distance(t.h, l2, v.fb[d]) : INFINITY;
                dd[d] = v.dblend ? blend_distance(t.h, l2, v.db[d]) : INFINITY;
            }
            float wf = fminf(dw[0], fminf(dw[1], dw[2])) > 0.0f ? 1.0f : 0.0f;
            float wd = fminf(dd[0], fminf(dd[1], dd[2])) > 0.0f ? 1.0f : 0.0f;
            if (wf != 0.0f && v.fblend)
#pragma unroll
                for (int d = 0; d < 3; ++d) wf = blend_factor(wf, dw[d], v.fr[d], v.fri[d]);
            if (wd != 0.0f && v.dblend)
#pragma unroll
                for (int d = 0; d < 3; ++d) wd = blend_factor(wd, dd[d], v.dr[d], v.dri[d]);
            fp_gather(sumD, wd);
            if (wf == 0.0f) continue;
            float val = 0.0f;  // outsideValueImg
            if (in) {
                const float q = trilinear(v, c, u, f);
                wide = wide || !(fabsf(q) <= FLT_MAX);
                val = fmaxf(1.0f, q);  // minValueImg
            }
            const FPair q = fp_prod(val, wf);
            fp_gather(sumI, q.h);
            sumI.l = __fadd_rn(sumI.l, q.l);
            fp_gather(sumW, wf);
        }
        float im = 0.0f;
        if (sumW.h > 0.0f) {
            // sumI / sumW: the float quotient and the correction by its residual
            const float q = __fdiv_rn(sumI.h, sumW.h);
            const float r = __fadd_rn(__fmaf_rn(-q, sumW.h, sumI.h), __fmaf_rn(-q, sumW.l, sumI.l));
            im = __fadd_rn(q, __fdividef(r, sumW.h));
        }
        wide = wide || !(fabsf(im) <= FLT_MAX);
        if (wide) d_wide[call % kWideCalls] = call;
        out_img[o0 + i] = wide ? NAN : im;
        out_w[o0 + i] = __fadd_rn(sumD.h, sumD.l);
    }
}

// The voxels that k_fuse_group of this call left as NaN, if it left any.
__global__ void __launch_bounds__(kFuseThreads)
    k_fuse_wide(const __grid_constant__ FuseViews fv, long long bx, long long by, long long bz, int nx, int ny, int nz,
                float *__restrict__ out_img, float *__restrict__ out_w, unsigned long long call)
{
    if (d_wide[call % kWideCalls] != call) return;
    const long long n = (long long)nx * ny * nz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (out_img[i] == out_img[i]) continue;
        const long long x = i % nx, y = i / nx % ny, z = i / nx / ny;
        fuse_voxel(fv, (double)(x + bx), (double)(y + by), (double)(z + bz), out_img[i], out_w[i]);
    }
}

thread_local std::string g_fuse_err;

int fuse_fail(int code, const std::string &m)
{
    g_fuse_err = m;
    return code;
}

}  // namespace
}  // namespace mvr

using namespace mvr;

extern "C" MVR_API const char *mvr_fuse_last_error(void) { return g_fuse_err.c_str(); }

extern "C" MVR_API int mvr_fuse_group(const mvr_fuse_view *views, int num_views, const long long bb_min[3],
                                      const int bb_dims[3], float *image_out, float *weight_out, int device,
                                      void *stream)
{
    if (!views || num_views < 1 || num_views > kFuseMaxViews || !bb_min || !bb_dims || !image_out || !weight_out)
        return fuse_fail(MVR_ERR_ARG, "mvr_fuse_group: 1..16 views, bounding box and outputs are required");
    for (int d = 0; d < 3; ++d)
        if (bb_dims[d] < 1) return fuse_fail(MVR_ERR_ARG, "mvr_fuse_group: empty bounding box");
    FuseViews fv{};
    fv.n = num_views;
    for (int k = 0; k < num_views; ++k) {
        const mvr_fuse_view &s = views[k];
        FuseView &v = fv.v[k];
        if (!s.img) return fuse_fail(MVR_ERR_ARG, "mvr_fuse_group: a view image is NULL");
        for (int d = 0; d < 3; ++d) {
            if (s.dims[d] < 2) return fuse_fail(MVR_ERR_ARG, "mvr_fuse_group: view sizes must be >= 2");
            v.dims[d] = s.dims[d];
            v.fb[d] = s.fusion_border[d];
            v.fr[d] = s.fusion_range[d];
            v.db[d] = s.decon_border[d];
            v.dr[d] = s.decon_range[d];
            v.fri[d] = 1.0f / v.fr[d];
            v.dri[d] = 1.0f / v.dr[d];
            v.top[d] = (float)(s.dims[d] - 1);
            v.half[d] = 0.5f * v.top[d];
        }
        v.fblend = s.fusion_blend;
        v.dblend = s.decon_blend;
        v.adjust = s.intensity_adjust ? 1 : 0;
        v.m00 = fp_from(s.intensity[0]);
        v.m01 = fp_from(s.intensity[1]);
        v.m[0] = s.intensity[0];
        v.m[1] = s.intensity[1];
        v.img = s.img;
        if (!invert_affine(s.model, v.inv)) return fuse_fail(MVR_ERR_ARG, "mvr_fuse_group: a view model is singular");
        for (int d = 0; d < 3; ++d) v.step[d] = fp_from(v.inv[4 * d]);
    }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fuse_fail(MVR_ERR_CUDA, cudaGetErrorString(e));
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    static std::atomic<unsigned long long> calls{0};
    const unsigned long long call = ++calls;
    const std::vector<FPair> &lut = blending_lut();
    e = cudaMemcpyToSymbolAsync(d_lut, lut.data(), sizeof(FPair) * lut.size(), 0, cudaMemcpyHostToDevice, s);
    // planes beyond the grid's y limit go out in further launches
    for (int z0 = 0; z0 < bb_dims[2] && e == cudaSuccess; z0 += 65535) {
        const int nz = std::min(65535, bb_dims[2] - z0);
        const long long at = (long long)z0 * bb_dims[0] * bb_dims[1];
        const int per = bb_dims[0] > kFuseLong ? 1 : kFuseRows;
        const dim3 grid((unsigned)((bb_dims[1] + per - 1) / per), (unsigned)nz);
        k_fuse_group<<<grid, kFuseThreads, 0, s>>>(fv, bb_min[0], bb_min[1], bb_min[2] + z0, bb_dims[0], bb_dims[1], nz,
                                                   image_out + at, weight_out + at, call);
        k_fuse_wide<<<152, kFuseThreads, 0, s>>>(fv, bb_min[0], bb_min[1], bb_min[2] + z0, bb_dims[0], bb_dims[1], nz,
                                                     image_out + at, weight_out + at, call);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fuse_fail(MVR_ERR_CUDA, std::string("mvr_fuse_group: ") + cudaGetErrorString(e));
    return MVR_OK;
}
