// y and z passes of the separable transforms (layout and tiles: sep.cuh), n = T V.
//
// A CTA takes 16 adjacent columns (one 128-byte line per transformed index).  With element
// i = t + T v (t < T, v < V):
//   phase 1, thread (column, t):  V-point DFT over v, straight from global memory (V loads of 8
//                                 bytes in flight per thread, a half-warp covers one line),
//                                 times W_n^(t k1), to shared memory at t + T k1;
//   phase 2, thread (column, k1): T-point DFT over t; position k2 + T k1 holds frequency
//                                 k1 + V k2, straight back to global memory.
// One exchange through shared memory per direction: a y pass has one, the z pass (forward,
// spectral product, inverse) two.  16 max(T, V) threads, so that one round covers either phase.
// Where a column's rows or planes are stored (mirrored, or a constant) is tabulated once per CTA as
// 32-bit byte offsets.  Bound by HBM and L2 traffic (y: 6.1 TB/s of algorithmic bytes on 288-long
// columns) and, in the z pass, by the load latency of the data and K^ (4.9 TB/s on 320).
#pragma once
#include "pdl.cuh"
#include "per_device.h"
#include "sep.cuh"
#include "sep_dft.cuh"

namespace mvr {

// Stored row or plane of domain index j, and whether it holds data.
struct SepRows {
    int lo, base, cnt, top;  // mirror: top = 2 N - 2
    int P, c;                // kernel
    __device__ __forceinline__ SepRows(const SepAxis &a, int map, int P_, int kd) : P(P_), c(kd / 2)
    {
        lo = a.lo;
        base = map == SEP_FILL ? a.q0 : a.v0;
        cnt = map == SEP_FILL ? a.nq : (map == SEP_MIRROR ? a.nv : kd);
        top = 2 * a.N - 2;
    }
    template <int MAP>
    __device__ __forceinline__ bool at(int j, int &i) const
    {
        if (MAP == SEP_MIRROR) {
            // one reflection suffices for every index that the result depends on; the others
            // (domain indices past the extension) read some stored row
            const int g = abs(lo + j);
            i = max(0, min(min(g, top - g) - base, cnt - 1));
            return true;
        }
        if (MAP == SEP_FILL) {
            i = lo + j - base;
        } else {
            i = j + c;
            if (i >= P) i -= P;
        }
        return (unsigned)i < (unsigned)cnt;
    }
};

template <int T, int V>
struct YzShape {
    static constexpr int n = T * V;
    static constexpr int W = T > V ? T : V;
    static constexpr int NT = 16 * W;
    // CTAs per SM the register budget is sized for
    static constexpr int TW = (n + NT - 1) / NT;  // twiddles a thread fetches
    // CTAs per SM the register budget is sized for: 1152 threads for the y passes (56 registers; 4-view
    // 256^3: 6.1 TB/s of algorithmic bytes, 5.0 at 640 threads), 960 for z (4.9 TB/s, 4.6 at 640); two
    // CTAs where a thread holds 24 values (56 registers spill: 5.5 -> 4.7 TB/s on 576-long columns)
    static constexpr int minb(int threads) { return W >= 24 ? 2 : (threads / NT > 8 ? 8 : threads / NT); }
    static constexpr int MINB_Y = minb(1152), MINB_Z = minb(960);
    // tile, twiddles, byte offsets of the input rows or planes
    static constexpr size_t smem = sizeof(float2) * (size_t)(16 * n + n) + sizeof(unsigned) * (size_t)n;
};

// Byte offsets of the stored rows (planes) of the domain indices, kSepNone for constant ones.
constexpr unsigned kSepNone = 0xffffffffu;
template <int n, int NT>
__device__ __forceinline__ void sep_offsets(unsigned *off, const SepRows &rows, int map, unsigned pitch)
{
    for (int j = threadIdx.x; j < n; j += NT) {
        int i;
        bool ok;
        if (map == SEP_MIRROR) ok = rows.at<SEP_MIRROR>(j, i);
        else if (map == SEP_FILL) ok = rows.at<SEP_FILL>(j, i);
        else ok = rows.at<SEP_KERNEL>(j, i);
        off[j] = ok ? (unsigned)i * pitch : kSepNone;
    }
}
// Phase 1's values of thread u: elements u + T v of the column at `base` + `at` bytes.
template <int T, int V>
__device__ __forceinline__ void sep_load(float2 (&a)[V], const float2 *base, unsigned at, const unsigned *off, int u,
                                         bool live, float2 fill)
{
    const char *p = reinterpret_cast<const char *>(base);
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const unsigned o = off[u + T * v];
        a[v] = live && o != kSepNone ? *reinterpret_cast<const float2 *>(p + (o + at)) : fill;
    }
}

// The twiddles: fetched ahead of the wait for the predecessor, put down behind the loads of the data.
template <int T, int V>
__device__ __forceinline__ void sep_tw_fetch(float2 (&r)[YzShape<T, V>::TW], const float2 *__restrict__ twg)
{
    typedef YzShape<T, V> SH;
#pragma unroll
    for (int k = 0; k < SH::TW; ++k) {
        const int i = threadIdx.x + k * SH::NT;
        r[k] = i < SH::n ? __ldg(&twg[i]) : make_float2(0.0f, 0.0f);
    }
}
template <int T, int V>
__device__ __forceinline__ void sep_tw_put(float2 *tw, const float2 (&r)[YzShape<T, V>::TW])
{
    typedef YzShape<T, V> SH;
#pragma unroll
    for (int k = 0; k < SH::TW; ++k) {
        const int i = threadIdx.x + k * SH::NT;
        if (i < SH::n) tw[i] = r[k];
    }
}

// ---- y forward, in place ----------------------------------------------------------------
// fill: value of the quotient's constant rows in column 0 (the x transform of ones: Px)
template <int T, int V>
__global__ void __launch_bounds__(YzShape<T, V>::NT, YzShape<T, V>::MINB_Y)
    k_sep_y_fwd(float2 *S, const SepTiles tl, SepGeom g, SepSlab sl, int map, int kdy, int kdz,
                const float2 *__restrict__ twg)
{
    typedef YzShape<T, V> SH;
    constexpr int n = SH::n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + 16 * n;
    // planes from the last to the first, all column blocks of a plane together: the rows pass before
    // left the last planes in L2
    const int z = gridDim.y - 1 - blockIdx.y, xb = sl.x0 + blockIdx.x;
    const SepTile &tile = tl.t[blockIdx.z];
    unsigned *off = reinterpret_cast<unsigned *>(tw + n);
    pdl_trigger();
    const int planes = map == SEP_MIRROR ? tile.a[2].nv : (map == SEP_FILL ? tile.a[2].nq : kdz);
    if (z >= planes) return;
    const SepRows rows(tile.a[1], map, n, kdy);
    float2 *base = S + (long long)blockIdx.z * g.stride;
    float2 *slot = base + ((long long)xb * g.Zs + z) * n * 16;
    const int c = threadIdx.x & 15, u = threadIdx.x >> 4;
    const float2 fill = make_float2(map == SEP_FILL && xb == 0 && c == 0 ? (float)g.P[0] : 0.0f, 0.0f);
    float2 twr[SH::TW];
    sep_tw_fetch<T, V>(twr, twg);
    sep_offsets<n, SH::NT>(off, rows, map, 128);
    __syncthreads();
    pdl_wait();
    float2 a[V];
    if (u < T) sep_load<T, V>(a, slot, 8 * c, off, u, true, fill);
    sep_tw_put<T, V>(tw, twr);
    __syncthreads();  // the twiddles; every row of the slot is read before phase 2 rewrites it
    if (u < T) {
        sep_dft<V, false>(a);
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], tw[u * k1]);
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) A[(u + T * k1) * 16 + c] = a[k1];
    }
    __syncthreads();
    float2 b[T];
    if (u < V) {
#pragma unroll
        for (int t = 0; t < T; ++t) b[t] = A[(t + T * u) * 16 + c];
        sep_dft<T, false>(b);
    }
    if (xb == 0) {
        // column 0 holds Z[k] = Y0[k] + i Ym[k]: Y0[k] = (Z[k] + conj Z[n-k]) / 2 stays, Ym[k] =
        // -i (Z[k] - conj Z[n-k]) / 2 goes to the Nyquist plane
        __syncthreads();
        if (u < V && c == 0)
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) A[u + V * k2] = b[k2];
        __syncthreads();
        if (u < V && c == 0) {
            float2 *nyq = base + (long long)g.nxb * g.Zs * n * 16 + (long long)z * n;
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) {
                const int f = u + V * k2;
                const float2 q = cconj(A[f == 0 ? 0 : n - f]);
                const float2 d = cscale(csub(b[k2], q), 0.5f);
                nyq[k2 + T * u] = make_float2(d.y, -d.x);
                b[k2] = cscale(cadd(b[k2], q), 0.5f);
            }
        }
    }
    if (u < V)
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) slot[(k2 + T * u) * 16 + c] = b[k2];
}

// ---- y inverse, in place ------------------------------------------------------------------
template <int T, int V>
__global__ void __launch_bounds__(YzShape<T, V>::NT, YzShape<T, V>::MINB_Y)
    k_sep_y_inv(float2 *S, const SepTiles tl, SepGeom g, SepSlab sl, int out_w, const float2 *__restrict__ twg)
{
    typedef YzShape<T, V> SH;
    constexpr int n = SH::n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + 16 * n;
    // column blocks from the last to the first: the z pass before left the last ones in L2
    const int z = blockIdx.x, xb = sl.x0 + gridDim.y - 1 - blockIdx.y;
    const SepTile &tile = tl.t[blockIdx.z];
    pdl_trigger();
    for (int i = threadIdx.x; i < n; i += SH::NT) tw[i] = __ldg(&twg[i]);
    if (z >= (out_w ? tile.a[2].nw : tile.a[2].nq)) return;
    const int r0 = out_w ? tile.a[1].w0 : tile.a[1].q0, nr = out_w ? tile.a[1].nw : tile.a[1].nq;
    const int off = tile.a[1].lo - r0;
    float2 *base = S + (long long)blockIdx.z * g.stride;
    float2 *slot = base + ((long long)xb * g.Zs + z) * n * 16;
    const int c = threadIdx.x & 15, u = threadIdx.x >> 4;
    pdl_wait();
    if (u < V) {
        float2 b[T];
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) b[k2] = slot[(k2 + T * u) * 16 + c];
        if (xb == 0 && c == 0) {  // column 0 back to Y0 + i Ym
            const float2 *nyq = base + (long long)g.nxb * g.Zs * n * 16 + (long long)z * n;
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) {
                const float2 ym = nyq[k2 + T * u];
                b[k2] = make_float2(b[k2].x - ym.y, b[k2].y + ym.x);
            }
        }
        sep_dft<T, true>(b);
#pragma unroll
        for (int t = 0; t < T; ++t) A[(t + T * u) * 16 + c] = b[t];
    }
    __syncthreads();
    if (u < T) {
        float2 a[V];
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) a[k1] = A[(u + T * k1) * 16 + c];
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], cconj(tw[u * k1]));
        sep_dft<V, true>(a);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int i = off + u + T * v;
            if ((unsigned)i < (unsigned)nr) slot[i * 16 + c] = a[v];
        }
    }
}

// ---- z: forward, times K, inverse -----------------------------------------------------------
template <int T, int V, bool MUL>
__global__ void __launch_bounds__(YzShape<T, V>::NT, YzShape<T, V>::MINB_Z)
    k_sep_z(const float2 *src, float2 *dst, const float2 *__restrict__ K, const SepTiles tl, SepGeom g,
            SepSlab sl, int map, int out_w, int kdz, const float2 *__restrict__ twg)
{
    typedef YzShape<T, V> SH;
    constexpr int n = SH::n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + 16 * n;
    unsigned *off = reinterpret_cast<unsigned *>(tw + n);
    const int Py = g.P[1];
    const SepTile &tile = tl.t[blockIdx.y];
    pdl_trigger();
    const int c = threadIdx.x & 15, u = threadIdx.x >> 4;
    // the 16 columns: one line of column block xb at y, or 16 y of the Nyquist plane (behind the
    // slab of column block 0)
    const int xq = blockIdx.x / Py, y = blockIdx.x - xq * Py;
    const bool nyq = xq == sl.n;
    const int xb = nyq ? g.nxb : sl.x0 + xq;
    const int cols = nyq ? min(16, Py - 16 * y) : 16;
    const bool live = c < cols;
    const unsigned pitch = nyq ? Py : Py * 16;
    const long long block = (long long)xb * Py * 16;  // times the planes of the buffer
    const unsigned at = 16 * y + c;
    const float2 *sp = src + (long long)blockIdx.y * g.stride + block * g.Zs;
    const SepRows rows(tile.a[2], map, n, kdz);
    // a plane of the constant quotient: its y transform is one value, at frequency 0 of column 0
    const float2 fill = make_float2(map == SEP_FILL && xb == 0 && y == 0 && c == 0
                                        ? (float)g.P[0] * (float)Py : 0.0f, 0.0f);
    float2 twr[SH::TW];
    sep_tw_fetch<T, V>(twr, twg);
    sep_offsets<n, SH::NT>(off, rows, map, 8 * pitch);
    __syncthreads();
    pdl_wait();
    float2 a[V];
    if (u < T) sep_load<T, V>(a, sp, 8 * at, off, u, live, fill);
    sep_tw_put<T, V>(tw, twr);
    __syncthreads();  // the twiddles
    if (u < T) {
        sep_dft<V, false>(a);
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], tw[u * k1]);
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) A[(u + T * k1) * 16 + c] = a[k1];
    }
    float2 b[T], kv[T];
    if (MUL && u < V) {  // K's values are on their way while the CTA meets at the barrier
        const float2 *kp = K + block * n;
        const unsigned k0 = at + T * u * pitch;
        const unsigned long long pol = sep_policy(g.stream);
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) kv[k2] = live ? sep_ldk(kp + (k0 + k2 * pitch), pol) : make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    if (u < V) {
#pragma unroll
        for (int t = 0; t < T; ++t) b[t] = A[(t + T * u) * 16 + c];
        sep_dft<T, false>(b);
    }
    if constexpr (!MUL) {  // a kernel spectrum: every plane of dst
        if (u < V && live) {
            float2 *dp = dst + block * n;
            const unsigned k0 = at + T * u * pitch;
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) dp[k0 + k2 * pitch] = b[k2];
        }
        return;
    } else {
        if (u < V) {
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) b[k2] = cmul(b[k2], kv[k2]);
            sep_dft<T, true>(b);
#pragma unroll
            for (int t = 0; t < T; ++t) A[(t + T * u) * 16 + c] = b[t];
        }
        __syncthreads();
        if (u < T && live) {
#pragma unroll
            for (int k1 = 0; k1 < V; ++k1) a[k1] = A[(u + T * k1) * 16 + c];
#pragma unroll
            for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], cconj(tw[u * k1]));
            sep_dft<V, true>(a);
            const int r0 = out_w ? tile.a[2].w0 : tile.a[2].q0, nr = out_w ? tile.a[2].nw : tile.a[2].nq;
            const int i0 = tile.a[2].lo - r0 + u;
            float2 *dp = dst + (long long)blockIdx.y * g.stride + block * g.Zs;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const unsigned i = i0 + T * v;
                if (i < (unsigned)nr) dp[at + i * pitch] = a[v];
            }
        }
    }
}

// The launches of one length.
struct YzOps {
    cudaError_t (*ready)();  // on the current device, before the first launch there
    cudaError_t (*y_fwd)(const SepGeom &, const SepSlab &, const SepTiles &, int, int, int, int, float2 *, const float2 *,
                         cudaStream_t, int);
    cudaError_t (*y_inv)(const SepGeom &, const SepSlab &, const SepTiles &, int, int, float2 *, const float2 *,
                         cudaStream_t, int);
    cudaError_t (*z)(const SepGeom &, const SepSlab &, const SepTiles &, int, int, int, int, const float2 *, float2 *,
                     const float2 *, const float2 *, cudaStream_t);
};

template <int T, int V>
struct Yz {
    typedef YzShape<T, V> SH;
    static cudaError_t limits()
    {
        const int m = (int)SH::smem;
        cudaError_t e = cudaFuncSetAttribute(k_sep_y_fwd<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sep_y_inv<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sep_z<T, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sep_z<T, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
        return e;
    }
    static cudaError_t ready()
    {
        static PerDevice once;
        return once(limits);
    }
    static cudaError_t y_fwd(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, int kdy, int kdz, float2 *S,
                             const float2 *tw, cudaStream_t s, int planes)
    {
        return launch_dep(sl.first, k_sep_y_fwd<T, V>, dim3(sl.n, planes, nt), SH::NT, SH::smem, s, S, tl, g, sl, map, kdy, kdz, tw);
    }
    static cudaError_t y_inv(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int out_w, float2 *S, const float2 *tw,
                             cudaStream_t s, int planes)
    {
        return launch_dep(sl.first, k_sep_y_inv<T, V>, dim3(planes, sl.n, nt), SH::NT, SH::smem, s, S, tl, g, sl, out_w, tw);
    }
    static cudaError_t z(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, int out_w, int kdz, const float2 *src,
                         float2 *dst, const float2 *K, const float2 *tw, cudaStream_t s)
    {
        const dim3 grid(sl.n * g.P[1] + (sl.x0 == 0 ? (g.P[1] + 15) / 16 : 0), nt);
        if (K)
            return launch_dep(sl.first, k_sep_z<T, V, true>, grid, SH::NT, SH::smem, s, src, dst, K, tl, g, sl, map, out_w, kdz, tw);
        return launch_dep(sl.first, k_sep_z<T, V, false>, grid, SH::NT, SH::smem, s, src, dst, K, tl, g, sl, map, out_w, kdz, tw);
    }
    static const YzOps *ops()
    {
        static const YzOps o = {&ready, &y_fwd, &y_inv, &z};
        return &o;
    }
};

// One per translation unit that instantiates lengths (NULL: not one of its own).
const YzOps *yz_ops_a(int n);
const YzOps *yz_ops_b(int n);
const YzOps *yz_ops_c(int n);
const YzOps *yz_ops_d(int n);

}  // namespace mvr
