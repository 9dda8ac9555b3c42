// x passes of the separable transforms (layout and tiles: sep.cuh): real rows of Px = 32 V, as
// m = 16 V packed complex values.
//
// A CTA of V warps takes 32 rows (consecutive stored rows y, then z).  Phase 1, item (row, t < 16):
// V-point DFT over the packed values t + 16 v, times W_m^(t k1); phase 2, item (row, k1): 16-point
// DFT over t, frequency k1 + V k2 at k2, fused with the packed-real split (which pairs f with
// m - f, held by item V - k1 of the same row: lanes 0-15 and 16-31 of one warp take the two, the
// values come over shuffles).  Item (row, k1) is one 128-byte line of column block k1, so shared
// memory holds [k1][row][16] with the rows padded to 144 bytes (16-byte accesses of 8 rows or of 8
// pieces of a row touch every bank once), and the lines move between shared and global memory
// 16 bytes a thread, 4 rows (512 contiguous bytes) a warp.
//
// Three to seven CTAs per SM, so that one CTA's loads overlap another's transforms: the
// passes are bound by instruction issue and HBM traffic together.
#pragma once
#include "pdl.cuh"
#include "rows_warp.cuh"
#include "sep.cuh"
#include "sep_dft.cuh"
#include "xy_plane.cuh"

namespace mvr {

constexpr int kSepRows = 32;  // rows per CTA
constexpr int kSepRS = 18;    // complex values per row of a column block in shared memory

template <int V>
struct SxShape {
    static constexpr int m = 16 * V, Px = 32 * V, NT = 32 * V;
    static constexpr int BS = kSepRows * kSepRS;  // complex values per column block
    static constexpr int MINB = NT > 512 ? 1 : (NT == 512 ? 2 : (896 / NT > 8 ? 8 : 896 / NT));
    static constexpr size_t smem = sizeof(float2) * (size_t)(V * BS + Px);
};

// Row tables of a CTA (static shared memory).
struct SxRows {
    long long a[kSepRows], b[kSepRows];  // row bases in the volume (-1: no row) and in the spectrum
};

// x phase 2 with the packed-real split (forward) or merge (inverse), one unit per warp.
template <int V, bool INV>
__device__ __forceinline__ void sx_p2(float2 *A, const float2 *twx)
{
    constexpr int T = 16;
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    int k1, row, h;
    bool self;
    if (V % 2 == 0) {  // pairs (1, V-1) ... and last (0, V/2), 16 rows each
        const int jp = w >> 1;
        h = l >> 4;
        row = (w & 1) * 16 + (l & 15);
        self = jp == V / 2 - 1;
        k1 = self ? (h ? V / 2 : 0) : (h ? V - 1 - jp : 1 + jp);
    } else {  // pairs (1, V-1) ... on 16 rows, and k1 = 0 on 32 rows
        self = w == V - 1;
        const int jp = w >> 1;
        h = self ? 0 : l >> 4;
        row = self ? l : (w & 1) * 16 + (l & 15);
        k1 = self ? 0 : (h ? V - 1 - jp : 1 + jp);
    }
    float4 *p = reinterpret_cast<float4 *>(A + k1 * SxShape<V>::BS + row * kSepRS);
    float2 b[T];
#pragma unroll
    for (int t = 0; t < T / 2; ++t) {
        const float4 q = p[t];
        b[2 * t] = make_float2(q.x, q.y);
        b[2 * t + 1] = make_float2(q.z, q.w);
    }
    if (!INV) sep_dft<T, false>(b);
    if (!self) {
#pragma unroll
        for (int k2 = 0; k2 < T / 2; ++k2) {
            const int k3 = T - 1 - k2;
            float2 ga, gb;
            ga.x = __shfl_xor_sync(0xffffffffu, b[k3].x, 16);
            ga.y = __shfl_xor_sync(0xffffffffu, b[k3].y, 16);
            gb.x = __shfl_xor_sync(0xffffffffu, b[k2].x, 16);
            gb.y = __shfl_xor_sync(0xffffffffu, b[k2].y, 16);
            b[k2] = xy_split_one<V, 0, INV>(b[k2], ga, k1 + V * k2, twx);
            b[k3] = xy_split_one<V, 0, INV>(b[k3], gb, k1 + V * k3, twx);
        }
    } else if (h == 0) {  // k1 = 0: f = V k2 pairs with slot 16 - k2; slots 0 and 8 with themselves
        b[0] = xy_split_one<V, 0, INV>(b[0], b[0], 0, twx);
        b[8] = xy_split_one<V, 0, INV>(b[8], b[8], V * 8, twx);
#pragma unroll
        for (int k2 = 1; k2 < T / 2; ++k2) {
            const int k3 = T - k2;
            const float2 oa = xy_split_one<V, 0, INV>(b[k2], b[k3], V * k2, twx);
            b[k3] = xy_split_one<V, 0, INV>(b[k3], b[k2], V * k3, twx);
            b[k2] = oa;
        }
    } else {  // k1 = V / 2: slot k2 pairs with slot 15 - k2
#pragma unroll
        for (int k2 = 0; k2 < T / 2; ++k2) {
            const int k3 = T - 1 - k2;
            const float2 oa = xy_split_one<V, 0, INV>(b[k2], b[k3], V / 2 + V * k2, twx);
            b[k3] = xy_split_one<V, 0, INV>(b[k3], b[k2], V / 2 + V * k3, twx);
            b[k2] = oa;
        }
    }
    if (INV) sep_dft<T, true>(b);
#pragma unroll
    for (int t = 0; t < T / 2; ++t) p[t] = make_float4(b[2 * t].x, b[2 * t].y, b[2 * t + 1].x, b[2 * t + 1].y);
}

template <int V, bool INV>
__device__ __forceinline__ void sx_p1(float2 (&a)[V], const float2 *twx, int t)
{
    if (!INV) {
        sep_dft<V, false>(a);
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], twx[2 * t * k1]);
    } else {
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], cconj(twx[2 * t * k1]));
        sep_dft<V, true>(a);
    }
}

// The CTA's lines from shared memory to the spectrum, and back (cp.async).
template <int V>
__device__ __forceinline__ void sx_store_lines(float2 *S, long long bstride, const float2 *A, const long long *rowb)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = threadIdx.x + k * SxShape<V>::NT;
        const int q = i & 7, row = (i >> 3) & 31, k1 = i >> 8;
        if (rowb[row] >= 0)
            *reinterpret_cast<float4 *>(S + k1 * bstride + rowb[row] + 2 * q) =
                *reinterpret_cast<const float4 *>(A + k1 * SxShape<V>::BS + row * kSepRS + 2 * q);
    }
}
template <int V>
__device__ __forceinline__ void sx_load_lines(float2 *A, const float2 *S, long long bstride, const long long *rowb)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = threadIdx.x + k * SxShape<V>::NT;
        const int q = i & 7, row = (i >> 3) & 31, k1 = i >> 8;
        const bool ok = rowb[row] >= 0;
        const unsigned d = (unsigned)__cvta_generic_to_shared(A + k1 * SxShape<V>::BS + row * kSepRS + 2 * q);
        const float2 *s = S + (ok ? k1 * bstride + rowb[row] + 2 * q : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(s), "r"(ok ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// The two voxels at x = g, g + 1 of a volume row under the mirror-single extension.
__device__ __forceinline__ float2 sx_pair(const float *__restrict__ row, int g, int N, bool vec)
{
    if (g >= 0 && g + 1 < N) {
        if (vec) return __ldg(reinterpret_cast<const float2 *>(row + g));
        return make_float2(__ldg(row + g), __ldg(row + g + 1));
    }
    const int a = abs(g), b = abs(g + 1), top = 2 * N - 2;
    return make_float2(__ldg(row + min(max(min(a, top - a), 0), N - 1)), __ldg(row + min(max(min(b, top - b), 0), N - 1)));
}
// The same with zeros outside [x0, x0 + n).
__device__ __forceinline__ float2 sx_pair_zero(const float *__restrict__ row, int g, int x0, int n, bool vec)
{
    const bool i0 = (unsigned)(g - x0) < (unsigned)n, i1 = (unsigned)(g + 1 - x0) < (unsigned)n;
    if (i0 && i1 && vec) return __ldg(reinterpret_cast<const float2 *>(row + g));
    return make_float2(i0 ? __ldg(row + g) : 0.0f, i1 ? __ldg(row + g + 1) : 0.0f);
}

// Rows r0 + [0, 32) of `ny` rows x `nz` planes from (y0, z0): their bases in the volume and in
// the tile's spectrum.
__device__ __forceinline__ void sx_rows(SxRows &sr, const SepTile &t, int r0, int y0, int ny, int z0, int nz, int Py)
{
    if (threadIdx.x < kSepRows) {
        const int r = r0 + threadIdx.x, z = r / ny, y = r - z * ny;
        const bool ok = z < nz;
        sr.a[threadIdx.x] = ok ? ((long long)(z0 + z) * t.a[1].N + y0 + y) * t.a[0].N : -1;
        sr.b[threadIdx.x] = ok ? ((long long)z * Py + y) * 16 : -1;
    }
}

// ---- forward ------------------------------------------------------------------------------
template <int V>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB)
    k_sep_x_fwd(SepSrc src, float2 *__restrict__ S, const SepTiles tl, SepGeom g, int vec,
                const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows sr;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int ny = src.kernel ? src.kd[1] : t.a[1].nv, nz = src.kernel ? src.kd[2] : t.a[2].nv;
    const int r0 = blockIdx.x * kSepRows;
    if (r0 >= ny * nz) return;
    for (int i = threadIdx.x; i < SH::Px; i += SH::NT) tw[i] = __ldg(&twg[i]);
    sx_rows(sr, t, r0, src.kernel ? 0 : t.a[1].v0, ny, src.kernel ? 0 : t.a[2].v0, nz, g.P[1]);
    __syncthreads();
    pdl_wait();
    for (int it = threadIdx.x; it < kSepRows * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long base = sr.a[row];
        float2 a[V];
        if (base < 0) {
#pragma unroll
            for (int v = 0; v < V; ++v) a[v] = make_float2(0.0f, 0.0f);
        } else if (!src.kernel) {
            const float *p = src.vol + base;
            const bool pv = vec && !((base + t.a[0].lo) & 1);
#pragma unroll
            for (int v = 0; v < V; ++v) a[v] = sx_pair(p, t.a[0].lo + 2 * (q + 16 * v), t.a[0].N, pv);
        } else {  // taps wrapped around the origin, scaled
            const int r = r0 + row, z = r / ny, y = r - z * ny;
            const float *p = src.vol + ((long long)z * src.kd[1] + y) * src.kd[0];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                float e[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int i = 2 * (q + 16 * v) + h + src.kd[0] / 2;
                    if (i >= SH::Px) i -= SH::Px;
                    e[h] = i < src.kd[0] ? (float)((double)p[i] * src.scale) : 0.0f;
                }
                a[v] = make_float2(e[0], e[1]);
            }
        }
        sx_p1<V, false>(a, tw, q);
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) A[k1 * SH::BS + row * kSepRS + q] = a[k1];
    }
    __syncthreads();
    sx_p2<V, false>(A, tw);
    __syncthreads();
    sx_store_lines<V>(S + (long long)blockIdx.y * g.stride, (long long)g.Zs * g.P[1] * 16, A, sr.b);
}

// ---- conv1 -> quotient -> forward ------------------------------------------------------------
// DeconvolutionMethods.java:71-74: img > 0 ? img / conv1 : 1, img zero outside the volume.
template <int V>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB)
    k_sep_x_ratio(float2 *__restrict__ S, const float *__restrict__ img, const SepTiles tl, SepGeom g, int vec,
                  const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows sr;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int r0 = blockIdx.x * kSepRows;
    if (r0 >= t.a[1].nq * t.a[2].nq) return;
    for (int i = threadIdx.x; i < SH::Px; i += SH::NT) tw[i] = __ldg(&twg[i]);
    sx_rows(sr, t, r0, t.a[1].q0, t.a[1].nq, t.a[2].q0, t.a[2].nq, g.P[1]);
    __syncthreads();
    pdl_wait();
    float2 *base = S + (long long)blockIdx.y * g.stride;
    const long long bstride = (long long)g.Zs * g.P[1] * 16;
    sx_load_lines<V>(A, base, bstride, sr.b);
    __syncthreads();
    sx_p2<V, true>(A, tw);
    __syncthreads();
    for (int it = threadIdx.x; it < kSepRows * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long ib = sr.a[row];
        const bool pv = vec && !((ib + t.a[0].lo) & 1);
        float2 im[V], a[V];
#pragma unroll
        for (int v = 0; v < V; ++v)
            im[v] = ib < 0 ? make_float2(0.0f, 0.0f)
                           : sx_pair_zero(img + ib, t.a[0].lo + 2 * (q + 16 * v), 0, t.a[0].N, pv);
        float2 *p = A + row * kSepRS + q;
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) a[k1] = p[k1 * SH::BS];
        sx_p1<V, true>(a, tw, q);
#pragma unroll
        for (int v = 0; v < V; ++v) a[v] = make_float2(quotient_fast(im[v].x, a[v].x), quotient_fast(im[v].y, a[v].y));
        sx_p1<V, false>(a, tw, q);
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) p[k1 * SH::BS] = a[k1];
    }
    __syncthreads();
    sx_p2<V, false>(A, tw);
    __syncthreads();
    sx_store_lines<V>(base, bstride, A, sr.b);
}

// ---- conv2 -> update ----------------------------------------------------------------------
// The written voxels alone: Seq (DeconvolutionMethods.java:103-182, 320-358) or the running product
// and final value of Mul (:370-419); with ST the change statistics over them.
template <int V, bool MUL, bool ST>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB)
    k_sep_x_update(const float2 *__restrict__ S, SepUpd u, int epi, const SepTiles tl, SepGeom g, int vec,
                   const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows sr;
    __shared__ double red_s[32], red_m[32];
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int r0 = blockIdx.x * kSepRows;
    const long long slot = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    if (r0 >= t.a[1].nw * t.a[2].nw) {
        if (ST && threadIdx.x == 0) {
            pdl_wait();  // the partials' last reader may still run
            u.partials[2 * slot] = 0.0;
            u.partials[2 * slot + 1] = -1.0;
        }
        return;
    }
    for (int i = threadIdx.x; i < SH::Px; i += SH::NT) tw[i] = __ldg(&twg[i]);
    sx_rows(sr, t, r0, t.a[1].w0, t.a[1].nw, t.a[2].w0, t.a[2].nw, g.P[1]);
    __syncthreads();
    pdl_wait();
    sx_load_lines<V>(A, S + (long long)blockIdx.y * g.stride, (long long)g.Zs * g.P[1] * 16, sr.b);
    __syncthreads();
    sx_p2<V, true>(A, tw);
    __syncthreads();
    float ksum = 0.0f, kcomp = 0.0f, kmax = -1.0f;
    const int x0 = t.a[0].w0, nx = t.a[0].nw;
    for (int it = threadIdx.x; it < kSepRows * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long vb = sr.a[row];
        if (vb < 0) continue;
        const bool pv = vec && !((vb + t.a[0].lo) & 1);
        const int g0 = t.a[0].lo + 2 * q;
        float2 last[V], wv[V], a[V];
        if (!MUL) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                last[v] = sx_pair_zero(u.psi + vb, g0 + 32 * v, x0, nx, pv);
                wv[v] = sx_pair_zero(u.weight[0] + vb, g0 + 32 * v, x0, nx, pv);
            }
        }
        const float2 *p = A + row * kSepRS + q;
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) a[k1] = p[k1 * SH::BS];
        sx_p1<V, true>(a, tw, q);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int x = g0 + 32 * v;
            const bool i0 = (unsigned)(x - x0) < (unsigned)nx, i1 = (unsigned)(x + 1 - x0) < (unsigned)nx;
            if (!i0 && !i1) continue;
            float next[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float cv = h ? a[v].y : a[v].x;
                if (!(h ? i1 : i0)) continue;
                float prev, w, f = cv;
                if (!MUL) {
                    prev = h ? last[v].y : last[v].x;
                    w = h ? wv[v].y : wv[v].x;
                } else {
                    float2 *pp = u.prod + vb + x + h;
                    if (epi == EPI_MUL_FIRST) {
                        *pp = mulprod_first(cv);
                        continue;
                    }
                    const float2 pr = u.nviews == 1 ? mulprod_first(cv) : mulprod_acc(*pp, cv);
                    if (epi == EPI_MUL_ACC) {
                        *pp = pr;
                        continue;
                    }
                    f = mulprod_root(pr, u.nviews);
                    w = 0.0f;
                    for (int k = 0; k < u.nviews; ++k) w += __ldg(u.weight[k] + vb + x + h);
                    w = w < 1.0f ? w : 1.0f;
                    prev = __ldg(u.psi + vb + x + h);
                }
                next[h] = MUL ? next_value(prev, f, w, u.c.two_lambda, u.c.tik, u.c.minI, u.c.maxI)
                              : next_value_fast(prev, f, w, u.c);
                if (ST) {
                    const float ch = next[h] - prev;  // signed change (DeconvolutionMethods.java:308)
                    const float ky = ch - kcomp;
                    const float kt = ksum + ky;
                    kcomp = (kt - ksum) - ky;
                    ksum = kt;
                    kmax = kmax > ch ? kmax : ch;
                }
            }
            if (MUL && epi != EPI_MUL_FINAL) continue;
            float *o = u.dst + vb + x;
            if (i0 && i1 && pv) {
                *reinterpret_cast<float2 *>(o) = make_float2(next[0], next[1]);
            } else {
                if (i0) o[0] = next[0];
                if (i1) o[1] = next[1];
            }
        }
    }
    if (ST) stats_to_partials(ksum, kcomp, kmax, red_s, red_m, u.partials, slot);
}

struct SxOps {
    cudaError_t (*fwd)(const SepGeom &, const SepTiles &, int, int, const SepSrc &, float2 *, int, const float2 *,
                       cudaStream_t);
    cudaError_t (*ratio)(const SepGeom &, const SepTiles &, int, int, const float *, float2 *, int, const float2 *,
                         cudaStream_t);
    cudaError_t (*update)(const SepGeom &, const SepTiles &, int, int, int, const SepUpd &, const float2 *, int,
                          const float2 *, cudaStream_t);
};

template <int V>
struct Sx {
    typedef SxShape<V> SH;
    static cudaError_t limits()
    {
        const int m = (int)SH::smem;
        cudaError_t e = cudaFuncSetAttribute(k_sep_x_fwd<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sep_x_ratio<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sep_x_update<V, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sep_x_update<V, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sep_x_update<V, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sep_x_update<V, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        return e;
    }
    static cudaError_t ready()
    {
        static const cudaError_t e = limits();
        return e;
    }
    static cudaError_t fwd(const SepGeom &g, const SepTiles &tl, int nt, int ctas, const SepSrc &src, float2 *S, int vec,
                           const float2 *tw, cudaStream_t s)
    {
        const cudaError_t e = ready();
        if (e != cudaSuccess) return e;
        return launch_pdl(k_sep_x_fwd<V>, dim3(ctas, nt), SH::NT, SH::smem, s, src, S, tl, g, vec, tw);
    }
    static cudaError_t ratio(const SepGeom &g, const SepTiles &tl, int nt, int ctas, const float *img, float2 *S,
                             int vec, const float2 *tw, cudaStream_t s)
    {
        const cudaError_t e = ready();
        if (e != cudaSuccess) return e;
        return launch_pdl(k_sep_x_ratio<V>, dim3(ctas, nt), SH::NT, SH::smem, s, S, img, tl, g, vec, tw);
    }
    static cudaError_t update(const SepGeom &g, const SepTiles &tl, int nt, int ctas, int epi, const SepUpd &u,
                              const float2 *S, int vec, const float2 *tw, cudaStream_t s)
    {
        const cudaError_t e = ready();
        if (e != cudaSuccess) return e;
        const dim3 grid(ctas, nt);
        const bool st = u.partials && (epi == EPI_SEQ || epi == EPI_MUL_FINAL);
#define SX_UPD(M, ST) launch_pdl(k_sep_x_update<V, M, ST>, grid, SH::NT, SH::smem, s, S, u, epi, tl, g, vec, tw)
        if (epi == EPI_SEQ) return st ? SX_UPD(false, true) : SX_UPD(false, false);
        return st ? SX_UPD(true, true) : SX_UPD(true, false);
#undef SX_UPD
    }
    static const SxOps *ops()
    {
        static const SxOps o = {&fwd, &ratio, &update};
        return &o;
    }
};

const SxOps *sx_ops_a(int n);
const SxOps *sx_ops_b(int n);
const SxOps *sx_ops_c(int n);

}  // namespace mvr
