// x passes of the separable transforms (layout and tiles: sep.cuh): real rows of Px = 32 V, as
// m = 16 V packed complex values.
//
// A CTA takes 32 or 16 rows (consecutive stored rows y, then z).  Phase 1, item (row, t < 16):
// V-point DFT over the packed values t + 16 v, times W_m^(t k1); phase 2, item (row, k1): 16-point
// DFT over t, frequency k1 + V k2 at k2, fused with the packed-real split (which pairs f with
// m - f, held by item V - k1 of the same row: lanes 0-15 and 16-31 of one warp take the two, the
// values come over shuffles).  Item (row, k1) is one 128-byte line of column block k1, so shared
// memory holds [k1][row][16] with the rows padded to 144 bytes (16-byte accesses of 8 rows or of 8
// pieces of a row touch every bank once), and the lines move between shared and global memory
// 16 bytes a thread, 4 rows (512 contiguous bytes) a warp.
//
// Three or more CTAs per SM, so that one CTA's loads overlap another's transforms: the passes are
// bound by instruction issue and HBM traffic together.  65536 rows of 288 reals (one view of 256^3),
// algorithmic bytes: forward 37 us (3.9 TB/s), quotient 56 us (3.9 TB/s), update 61 us (4.5 TB/s).
#pragma once
#include "pdl.cuh"
#include "per_device.h"
#include "rows_warp.cuh"
#include "sep.cuh"
#include "sep_dft.cuh"
#include "xy_plane.cuh"

namespace mvr {

constexpr int kSepRS = 18;  // complex values per row of a column block in shared memory

// 32 rows and a warp per phase-2 unit up to V = 10; 16 rows above (half the shared memory and twice
// the CTAs per SM for the same threads), with 256 threads for V = 12 ... 16 so that phase 1 is
// one full round.
template <int V>
struct SxShape {
    static constexpr int m = 16 * V, Px = 32 * V;
    static constexpr int R = V >= 12 ? 16 : 32;  // rows per CTA
    static constexpr int NT = V >= 12 && V <= 16 ? 256 : R * V;
    static constexpr int BS = R * kSepRS;        // complex values per column block
    static constexpr int UNITS = V * R / 32;     // phase-2 units of a warp each
    // CTAs per SM for a register budget sized to `threads` threads per SM
    static constexpr int minb(int threads) { return NT > threads ? 1 : (threads / NT > 8 ? 8 : threads / NT); }
    // measured on 65536 rows of 288 (4-view 256^3) and of 576: forward 37.6 us at 1152 (40.7 at 896),
    // quotient 53.7 us at 896 (56.2 at 1152), Seq update 60 us at 896 (75 at 1152); update of the
    // lengths that load a chunk at a time, 285 us at 1152 (361 at 896)
    static constexpr int MINB_FWD = minb(1152), MINB_RATIO = minb(896), MINB_UPD = minb(V < 12 ? 896 : 1152);
    static constexpr size_t smem = sizeof(float2) * (size_t)(V * BS + Px);
};

// Row tables of a CTA (static shared memory).
template <int V>
struct SxRows {
    long long a[SxShape<V>::R], b[SxShape<V>::R];  // row bases in the volume (-1: no row) and in the spectrum
    unsigned flag;                                 // blocks are marked (BadMap)
};

// x phase 2 with the packed-real split (forward) or merge (inverse), one unit per warp and round.
template <int V, bool INV>
__device__ __forceinline__ void sx_p2(float2 *A, const float2 *twx)
{
    constexpr int T = 16, RB = SxShape<V>::R / 16;
    const int l = threadIdx.x & 31;
    for (int w = threadIdx.x >> 5; w < SxShape<V>::UNITS; w += SxShape<V>::NT / 32) {
    int k1, row, h;
    bool self;
    if (V % 2 == 0) {  // pairs (1, V-1) ... and last (0, V/2), 16 rows each
        const int jp = w / RB;
        h = l >> 4;
        row = (w % RB) * 16 + (l & 15);
        self = jp == V / 2 - 1;
        k1 = self ? (h ? V / 2 : 0) : (h ? V - 1 - jp : 1 + jp);
    } else {  // pairs (1, V-1) ... on 16 rows, and k1 = 0 on 32 rows
        static_assert(V % 2 == 0 || RB == 2, "odd V: 32 rows");
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
}

// Twiddles in shared memory: W_Px^f for the split (f < m), then W_m^(t k1) at m + 16 k1 + t, so that
// the 16 lanes of a row read one line (W_Px^(2 t k1) from the plain table is up to a 16-way bank
// conflict: forward 40.8 -> 37.6 us, quotient 55.6 -> 53.7 us on 65536 rows of 288, forward 135 -> 115 us
// on the rows of 576 of a 512 x 512 x 256 view).
template <int V>
__device__ __forceinline__ void sx_twiddles(float2 *tw, const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    for (int i = threadIdx.x; i < SH::m; i += SH::NT) {
        tw[i] = __ldg(&twg[i]);
        tw[SH::m + i] = __ldg(&twg[2 * (i & 15) * (i >> 4)]);
    }
}

template <int V, bool INV>
__device__ __forceinline__ void sx_p1(float2 (&a)[V], const float2 *twx, int t)
{
    const float2 *w = twx + SxShape<V>::m + t;
    if (!INV) {
        sep_dft<V, false>(a);
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], w[16 * k1]);
    } else {
#pragma unroll
        for (int k1 = 1; k1 < V; ++k1) a[k1] = cmul(a[k1], cconj(w[16 * k1]));
        sep_dft<V, true>(a);
    }
}

// The CTA's lines between shared memory and the spectrum: a thread keeps its 16-byte piece q of a
// row and walks the column blocks (one pointer step each).  f(shared piece, global piece, row
// exists), the row's base checked once per row.
template <int V, class F>
__device__ __forceinline__ void sx_lines(float2 *A, float2 *S, long long bstride, const long long *rowb, F f)
{
    typedef SxShape<V> SH;
    constexpr int per = 8 * SH::R;                            // pieces per column block
    constexpr int G = SH::NT >= per ? SH::NT / per : 1;       // column blocks at a time
    constexpr int step = SH::NT >= per ? SH::R : SH::NT / 8;  // rows at a time
    const int tid = threadIdx.x;
    if (G * per < SH::NT && tid >= G * per) return;
    const int g = G > 1 ? tid / per : 0, q = tid & 7;
#pragma unroll
    for (int r0 = 0; r0 < SH::R; r0 += step) {
        const int row = r0 + ((tid - g * per) >> 3);
        if (SH::R % step != 0 && row >= SH::R) break;
        const long long rb = rowb[row];
        float2 *a = A + g * SH::BS + row * kSepRS + 2 * q;
        float2 *p = S + (rb >= 0 ? rb + 2 * q + g * bstride : 0);
#pragma unroll
        for (int k1 = 0; k1 < V; k1 += G) {
            if (V % G == 0 || k1 + g < V) f(a + k1 * SH::BS, p, rb >= 0);
            p += rb >= 0 ? G * bstride : 0;
        }
    }
}
template <int V>
__device__ __forceinline__ void sx_store_lines(float2 *S, long long bstride, float2 *A, const long long *rowb)
{
    sx_lines<V>(A, S, bstride, rowb, [](float2 *a, float2 *p, bool ok) {
        if (ok) *reinterpret_cast<float4 *>(p) = *reinterpret_cast<const float4 *>(a);
    });
}
template <int V>
__device__ __forceinline__ void sx_load_lines(float2 *A, const float2 *S, long long bstride, const long long *rowb)
{
    sx_lines<V>(A, const_cast<float2 *>(S), bstride, rowb, [](float2 *a, float2 *p, bool ok) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(a);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(ok ? 16 : 0) : "memory");
    });
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Pairs of voxels (x, x + 1) of a volume row at x = g0 + 32 v, v < V, with zeros outside
// [x0, x0 + n).  PAIRS: no pair is split by the range and every row starts on 8 bytes, so that a
// pair is one predicated 8-byte load.
template <int V, bool PAIRS>
__device__ __forceinline__ void sx_load_zero(float2 (&a)[V], const float *row, int g0, int x0, int n,
                                             unsigned long long pol)
{
    const float *p = row + g0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int r = g0 - x0 + 32 * v;
        if (PAIRS) {
            a[v] = (unsigned)r < (unsigned)n ? sep_ld2(p + 32 * v, pol) : make_float2(0.0f, 0.0f);
        } else {
            a[v].x = (unsigned)r < (unsigned)n ? sep_ld(p + 32 * v, pol) : 0.0f;
            a[v].y = (unsigned)(r + 1) < (unsigned)n ? sep_ld(p + 32 * v + 1, pol) : 0.0f;
        }
    }
}
// The same under the mirror-single extension of [0, N), no voxel beyond `last` (the last one that the tile
// takes from psi: a domain that is longer would hold the magnitudes of others).
template <int V, bool PAIRS>
__device__ __forceinline__ void sx_load_mirror(float2 (&a)[V], const float *row, int g0, int N, int last,
                                               unsigned long long pol)
{
    const float *p = row + g0;
    const int top = 2 * N - 2;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int g = g0 + 32 * v;
        if (PAIRS && (unsigned)g < (unsigned)last) {
            a[v] = sep_ld2(p + 32 * v, pol);
        } else {
            const int i = abs(g), j = abs(g + 1);
            a[v].x = sep_ld(row + min(max(min(i, top - i), 0), last), pol);
            a[v].y = sep_ld(row + min(max(min(j, top - j), 0), last), pol);
        }
    }
}
// Pairs start at even offsets from an even lo: whole in [x0, x0 + n) and 8-byte aligned in every row?
__device__ __forceinline__ bool sx_pairs(int vec, const SepAxis &a, int x0, int n)
{
    return vec && !((a.N | a.lo | x0 | n) & 1);
}

// Rows r0 + [0, R) of `ny` rows x `nz` planes from (y0, z0): their bases in the volume and in
// the tile's spectrum.
template <int V>
__device__ __forceinline__ void sx_rows(SxRows<V> &sr, const SepTile &t, int r0, int y0, int ny, int z0, int nz, int Py)
{
    if (threadIdx.x < SxShape<V>::R) {
        const int r = r0 + threadIdx.x, z = r / ny, y = r - z * ny;
        const bool ok = z < nz;
        sr.a[threadIdx.x] = ok ? ((long long)(z0 + z) * t.a[1].N + y0 + y) * t.a[0].N : -1;
        sr.b[threadIdx.x] = ok ? ((long long)z * Py + y) * 16 : -1;
    }
}

// The quotient by a quarter of conv1 (K1^ carries the factor): the approximate division takes divisors up to
// 2^126 and returns 0 beyond.  Its two ulp are not seen behind the transforms' rounding: with IEEE divisions
// and roots here and in the update the errors against 64 bits stay where they are (156 x 156 x 124 block
// 1.1e-7 and 1.2e-7, 2 views of 128 x 128 x 64 6.5e-7 and 6.6e-7, 256^3 1.3e-7 both) and 4 views of 256^3 take 2 to
// 8 % longer.
__device__ __forceinline__ float sx_quotient(float img, float quarter)
{
    return img > 0.0f ? __fdividef(0.25f * img, quarter) : 1.0f;
}

// ---- values that are not finite (BadMap) ----------------------------------------------------
// A row item whose phase-1 transform shows one (its zero frequency is the sum of the inputs) is done
// again by the thread that had it, with 1 in the value's place, as plain sums: the ordinary path pays two
// comparisons per item and one register.  (No local arrays and no calls: with either, the kernel has a stack,
// and 2 views of 128 x 128 x 64 take 4 % longer; so 1.5 %, 4 views of 256^3 0.8 %.)
__device__ __forceinline__ bool sx_finite(float v) { return fabsf(v) <= 3.402823466e38f; }
__device__ __forceinline__ bool sx_finite(float2 v) { return sx_finite(v.x) && sx_finite(v.y); }

// The word at m (or 0) into shared memory, its way there behind the loads that f starts and waits for.
template <class F>
__device__ __forceinline__ void sx_flag(unsigned &flag, const unsigned *m, F f)
{
    const unsigned v = threadIdx.x == 0 && m ? *m : 0;
    f();
    if (threadIdx.x == 0) flag = v;
}

template <int V>
__device__ __forceinline__ float2 sx_root(const float2 *tw, int j)  // W_V^j, j < V^2
{
    const int f = 32 * (j % V), m = SxShape<V>::m;
    return f < m ? tw[f] : make_float2(-tw[f - m].x, -tw[f - m].y);
}
// Phase 1 of x(v), v < V, into the item's line elements p[k1 BS].
template <int V, class X>
__device__ __forceinline__ void sx_p1_sums(float2 *p, const float2 *tw, int t, X x)
{
#pragma unroll 1
    for (int k1 = 0; k1 < V; ++k1) {
        float2 s = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int v = 0; v < V; ++v) s = cadd(s, cmul(x(v), sx_root<V>(tw, v * k1)));
        p[k1 * SxShape<V>::BS] = cmul(s, tw[SxShape<V>::m + 16 * k1 + t]);
    }
}
// psi: the item at x = g0 + 32 v + {0, 1} of the row at (y, z)
template <int V>
__device__ __forceinline__ void sx_fwd_again(BadMap *b, const float *row, float2 *p, const float2 *tw, int t, int g0, int N,
                                             int last, int y, int z)
{
    sx_p1_sums<V>(p, tw, t, [&](int v) {
        float c[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = abs(g0 + 32 * v + h), j = min(max(min(i, 2 * N - 2 - i), 0), last);
            c[h] = row[j];
            if (sx_finite(c[h])) continue;
            bad_mark(b, BAD_PSI, j, y, z);
            c[h] = 1.0f;
        }
        return make_float2(c[0], c[1]);
    });
}
// The quotient, conv1's phase-1 values still in p; s[v stride]: the item's elements of the spectrum lines,
// which the CTA has read and not yet written.
template <int V>
__device__ __forceinline__ void sx_ratio_again(BadMap *b, const float *row, float2 *p, float2 *s, long long stride,
                                               const float2 *tw, int t, int g0, int N, int y, int z)
{
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
        float2 q = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int k1 = 0; k1 < V; ++k1)
            q = cadd(q, cmul(p[k1 * SxShape<V>::BS], cconj(cmul(tw[SxShape<V>::m + 16 * k1 + t], sx_root<V>(tw, v * k1)))));
        float c[2] = {q.x, q.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = g0 + 32 * v + h;
            const bool in = i >= 0 && i < N;
            c[h] = sx_quotient(in ? row[i] : 0.0f, c[h]);
            if (sx_finite(c[h])) continue;
            if (in) bad_mark(b, BAD_QUOTIENT, i, y, z);
            c[h] = 1.0f;
        }
        s[v * stride] = make_float2(c[0], c[1]);
    }
    sx_p1_sums<V>(p, tw, t, [&](int v) { return s[v * stride]; });
}

// ---- forward ------------------------------------------------------------------------------
template <int V>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB_FWD)
    k_sep_x_fwd(SepSrc src, float2 *__restrict__ S, const SepTiles tl, SepGeom g, int vec,
                const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows<V> sr;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int ny = src.kernel ? src.kd[1] : t.a[1].nv, nz = src.kernel ? src.kd[2] : t.a[2].nv;
    const int r0 = blockIdx.x * SH::R;
    if (r0 >= ny * nz) return;
    sx_twiddles<V>(tw, twg);
    sx_rows<V>(sr, t, r0, src.kernel ? 0 : t.a[1].v0, ny, src.kernel ? 0 : t.a[2].v0, nz, g.P[1]);
    __syncthreads();
    const unsigned long long pol = sep_policy(g.stream);
    const bool pairs = sx_pairs(vec, t.a[0], 0, t.a[0].N);
    unsigned again = 0;  // bit k: the thread's k-th item
    pdl_wait();
    if ((g.clear & 1) && blockIdx.x + blockIdx.y + threadIdx.x == 0) bad_clear(g.bad, BAD_QUOTIENT);
    for (int it = threadIdx.x; it < SH::R * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long base = sr.a[row];
        float2 a[V];
        if (base < 0) {
#pragma unroll
            for (int v = 0; v < V; ++v) a[v] = make_float2(0.0f, 0.0f);
        } else if (!src.kernel) {
            const float *p = src.vol + base;
            const int last = t.a[0].v0 + t.a[0].nv - 1;
            if (pairs) sx_load_mirror<V, true>(a, p, t.a[0].lo + 2 * q, t.a[0].N, last, pol);
            else sx_load_mirror<V, false>(a, p, t.a[0].lo + 2 * q, t.a[0].N, last, pol);
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
        if (!sx_finite(a[0])) again |= 1u << it / SH::NT;
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) A[k1 * SH::BS + row * kSepRS + q] = a[k1];
    }
    if (again && g.bad)
#pragma unroll 1
        for (int it = threadIdx.x; it < SH::R * 16; it += SH::NT) {
            if (!(again >> it / SH::NT & 1)) continue;
            const int q = it & 15, row = it >> 4, r = r0 + row;
            sx_fwd_again<V>(g.bad, src.vol + sr.a[row], A + row * kSepRS + q, tw, q, t.a[0].lo + 2 * q, t.a[0].N,
                            t.a[0].v0 + t.a[0].nv - 1, t.a[1].v0 + r % ny, t.a[2].v0 + r / ny);
        }
    __syncthreads();
    sx_p2<V, false>(A, tw);
    __syncthreads();
    sx_store_lines<V>(S + (long long)blockIdx.y * g.stride, (long long)g.Zs * g.P[1] * 16, A, sr.b);
}

// ---- conv1 -> quotient -> forward ------------------------------------------------------------
// DeconvolutionMethods.java:71-74: img > 0 ? img / conv1 : 1, img zero outside the volume.
template <int V>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB_RATIO)
    k_sep_x_ratio(float2 *__restrict__ S, const float *__restrict__ img, const SepTiles tl, SepGeom g, int vec,
                  const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows<V> sr;
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int r0 = blockIdx.x * SH::R;
    if (r0 >= t.a[1].nq * t.a[2].nq) return;
    sx_twiddles<V>(tw, twg);
    sx_rows<V>(sr, t, r0, t.a[1].q0, t.a[1].nq, t.a[2].q0, t.a[2].nq, g.P[1]);
    __syncthreads();
    pdl_wait();
    float2 *base = S + (long long)blockIdx.y * g.stride;
    const long long bstride = (long long)g.Zs * g.P[1] * 16;
    const unsigned long long pol = sep_policy(g.stream);
    const int end = t.a[0].v0 + t.a[0].nv;  // no image beyond the tile's psi: N, or the end of a dim block
    const bool pairs = sx_pairs(vec, t.a[0], 0, end);
    unsigned again = 0;
    sx_flag(sr.flag, g.bad ? &g.bad->any[BAD_PSI] : nullptr, [&] { sx_load_lines<V>(A, base, bstride, sr.b); });
    __syncthreads();
    sx_p2<V, true>(A, tw);
    __syncthreads();
    for (int it = threadIdx.x; it < SH::R * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long ib = sr.a[row];
        constexpr bool EARLY = V < 12;  // the image ahead of the transform, as the registers allow
        float2 im[V], a[V];
        const int n = ib < 0 ? 0 : end;  // no row: no voxel
        if (EARLY) {
            if (pairs) sx_load_zero<V, true>(im, img + ib, t.a[0].lo + 2 * q, 0, n, pol);
            else sx_load_zero<V, false>(im, img + ib, t.a[0].lo + 2 * q, 0, n, pol);
        }
        float2 *p = A + row * kSepRS + q;
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) a[k1] = p[k1 * SH::BS];
        sx_p1<V, true>(a, tw, q);
        if (!EARLY) {
            if (pairs) sx_load_zero<V, true>(im, img + ib, t.a[0].lo + 2 * q, 0, n, pol);
            else sx_load_zero<V, false>(im, img + ib, t.a[0].lo + 2 * q, 0, n, pol);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) a[v] = make_float2(sx_quotient(im[v].x, a[v].x), sx_quotient(im[v].y, a[v].y));
        sx_p1<V, false>(a, tw, q);
        if (g.bad && !sx_finite(a[0])) {
            again |= 1u << it / SH::NT;
            continue;
        }
#pragma unroll
        for (int k1 = 0; k1 < V; ++k1) p[k1 * SH::BS] = a[k1];
    }
    if (again)
#pragma unroll 1
        for (int it = threadIdx.x; it < SH::R * 16; it += SH::NT) {
            if (!(again >> it / SH::NT & 1)) continue;
            const int q = it & 15, row = it >> 4, r = r0 + row;
            if (sr.a[row] < 0) continue;
            sx_ratio_again<V>(g.bad, img + sr.a[row], A + row * kSepRS + q, base + sr.b[row] + q, bstride, tw, q,
                              t.a[0].lo + 2 * q, end, t.a[1].q0 + r % t.a[1].nq, t.a[2].q0 + r / t.a[1].nq);
        }
    if (sr.flag) {  // the quotients of a block that reads it, where the image is positive
        const int N = t.a[0].N;
#pragma unroll 1
        for (int i = threadIdx.x; i < SH::R * N; i += SH::NT) {
            const int row = i / N, x = i - row * N, r = r0 + row;
            if (sr.a[row] >= 0 && img[sr.a[row] + x] > 0.0f)
                bad_mark(g.bad, BAD_QUOTIENT, x, t.a[1].q0 + r % t.a[1].nq, t.a[2].q0 + r / t.a[1].nq, true);
        }
    }
    __syncthreads();
    sx_p2<V, false>(A, tw);
    __syncthreads();
    sx_store_lines<V>(base, bstride, A, sr.b);
}

// ---- conv2 -> update ----------------------------------------------------------------------
__device__ __forceinline__ void sx_change(float next, float last, float &ksum, float &kcomp, float &kmax)
{
    const float ch = next - last;  // signed change (DeconvolutionMethods.java:308)
    const float ky = ch - kcomp;
    const float kt = ksum + ky;
    kcomp = (kt - ksum) - ky;
    ksum = kt;
    kmax = kmax > ch ? kmax : ch;
}

// One row item of the Seq update: conv2 at the voxels x = g0 + 32 v + {0, 1}, the new psi for those
// in [x0, x0 + nx).
template <int V, bool ST, bool PAIRS>
__device__ __forceinline__ void sx_update_row(const float2 *p, const float2 *tw, int q, const SepUpd &u, long long vb,
                                              int g0, int x0, int nx, float &ksum, float &kcomp, float &kmax,
                                              unsigned long long pol)
{
    constexpr int BS = SxShape<V>::BS;
    // psi and the weight ahead of the transform where the registers allow, else 6 pairs at a time, all
    // loads of a chunk ahead of its stores (a load per store, in turn: 1.71 against 1.37 ms for the 6
    // views of 512 x 512 x 256)
    constexpr bool EARLY = V < 12;
    constexpr int CH = EARLY ? V : 6;
    float2 prev[CH], w[CH], a[V];
    if (EARLY) {
        sx_load_zero<CH, PAIRS>(prev, u.psi + vb, g0, x0, nx, pol);
        sx_load_zero<CH, PAIRS>(w, u.weight[0] + vb, g0, x0, nx, pol);
    }
#pragma unroll
    for (int k1 = 0; k1 < V; ++k1) a[k1] = p[k1 * BS];
    sx_p1<V, true>(a, tw, q);
#pragma unroll
    for (int c0 = 0; c0 < V; c0 += CH) {
        if (!EARLY) {  // (pairs past the last of a partial chunk lie past the tile, so past the range)
            sx_load_zero<CH, PAIRS>(prev, u.psi + vb, g0 + 32 * c0, x0, nx, pol);
            sx_load_zero<CH, PAIRS>(w, u.weight[0] + vb, g0 + 32 * c0, x0, nx, pol);
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int v = c0 + j;
            if (v >= V) break;
            const int r = g0 - x0 + 32 * v;
            const bool i0 = (unsigned)r < (unsigned)nx, i1 = PAIRS ? i0 : (unsigned)(r + 1) < (unsigned)nx;
            if (!i0 && !i1) continue;
            const float2 next = make_float2(next_value_fast(prev[j].x, a[v].x, w[j].x, u.c),
                                            next_value_fast(prev[j].y, a[v].y, w[j].y, u.c));
            if (ST && i0) sx_change(next.x, prev[j].x, ksum, kcomp, kmax);
            if (ST && i1) sx_change(next.y, prev[j].y, ksum, kcomp, kmax);
            float *o = u.dst + vb + g0 + 32 * v;
            if (PAIRS) {
                sep_st2(o, next, pol);
            } else {
                if (i0) sep_st(o, next.x, pol);
                if (i1) sep_st(o + 1, next.y, pol);
            }
        }
    }
}

// The Mul pass over the CTA's rows of conv2 (natural order in shared memory): the running product
// (EPI_MUL_FIRST, EPI_MUL_ACC) or the final value, U pairs of voxels a thread at a time with all
// their loads in flight; lanes run along x.  (On the registers of the transform, as Seq does it, the
// products spill or are loaded one by one: 82 us a view on 211 x 187 x 143, 49 us in this form.)
template <int V, bool ST>
__device__ __forceinline__ void sx_mul_rows(const float2 *A, const SepUpd &u, int epi, const SepTile &t,
                                            const long long *rowa, float &ksum, float &kcomp, float &kmax,
                                            unsigned long long pol)
{
    typedef SxShape<V> SH;
    constexpr int U = 4, items = SH::R * SH::m;
    const int lo = t.a[0].lo, x0 = t.a[0].w0, nx = t.a[0].nw;
    const bool acc = epi != EPI_MUL_FIRST && u.nviews > 1, fin = epi == EPI_MUL_FINAL;
    for (int i0 = threadIdx.x; i0 < items; i0 += U * SH::NT) {
        float2 pr[U][2], last[U], w[U];
        long long at[U];
        bool in[U][2];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * SH::NT, row = i / SH::m, j = i - row * SH::m;
            const long long vb = i < items ? rowa[row] : -1;
            const int r = lo + 2 * j - x0;
            in[k][0] = vb >= 0 && (unsigned)r < (unsigned)nx;
            in[k][1] = vb >= 0 && (unsigned)(r + 1) < (unsigned)nx;
            at[k] = vb + lo + 2 * j;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                pr[k][h] = acc && in[k][h] ? u.prod[at[k] + h] : make_float2(0.0f, 0.0f);
            last[k] = w[k] = make_float2(0.0f, 0.0f);
            if (fin) {
                if (in[k][0]) last[k].x = sep_ld(u.psi + at[k], pol);
                if (in[k][1]) last[k].y = sep_ld(u.psi + at[k] + 1, pol);
            }
        }
        if (fin)
            for (int v = 0; v < u.nviews; ++v) {
                float2 wv[U];
#pragma unroll
                for (int k = 0; k < U; ++k)
                    wv[k] = make_float2(in[k][0] ? sep_ld(u.weight[v] + at[k], pol) : 0.0f,
                                        in[k][1] ? sep_ld(u.weight[v] + at[k] + 1, pol) : 0.0f);
#pragma unroll
                for (int k = 0; k < U; ++k) w[k] = cadd(w[k], wv[k]);
            }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + k * SH::NT, row = i / SH::m, j = i - row * SH::m;
            if (i >= items) break;
            const float2 c = A[(j >> 4) * SH::BS + row * kSepRS + (j & 15)];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!in[k][h]) continue;
                const float cv = h ? c.y : c.x;
                const float2 q = acc ? mulprod_acc(pr[k][h], cv) : mulprod_first(cv);
                if (!fin) {
                    u.prod[at[k] + h] = q;
                    continue;
                }
                const float wt = h ? w[k].y : w[k].x, prev = h ? last[k].y : last[k].x;
                const float next = next_value(prev, mulprod_root(q, u.nviews), wt < 1.0f ? wt : 1.0f, u.c.two_lambda,
                                              u.c.tik, u.c.minI, u.c.maxI);
                if (ST) sx_change(next, prev, ksum, kcomp, kmax);
                sep_st(u.dst + at[k] + h, next, pol);
            }
        }
    }
}

// psi of voxel `at` in a block whose second convolution is NaN: next_value takes minI.
__device__ __forceinline__ void sx_bad_value(const SepUpd &u, bool mul, long long at)
{
    float w = 0.0f;
    for (int v = 0; v < u.nviews; ++v) w += u.weight[v][at];
    if (mul) w = w < 1.0f ? w : 1.0f;
    const float last = u.psi[at];
    u.dst[at] = __fadd_rn(last, __fmul_rn(__fsub_rn(u.c.minI, last), w));
}

// The written voxels alone: Seq (DeconvolutionMethods.java:103-182, 320-358) or the running product
// and final value of Mul (:370-419); with ST the change statistics over them.
template <int V, bool MUL, bool ST>
__global__ void __launch_bounds__(SxShape<V>::NT, SxShape<V>::MINB_UPD)
    k_sep_x_update(const float2 *__restrict__ S, SepUpd u, int epi, const SepTiles tl, SepGeom g, int vec,
                   const float2 *__restrict__ twg)
{
    typedef SxShape<V> SH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SxRows<V> sr;
    __shared__ double red_s[32], red_m[32];
    float2 *A = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = A + V * SH::BS;
    const SepTile &t = tl.t[blockIdx.y];
    pdl_trigger();
    const int r0 = blockIdx.x * SH::R;
    const long long slot = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    if (r0 >= t.a[1].nw * t.a[2].nw) {
        if (ST && threadIdx.x == 0) {
            pdl_wait();  // the partials' last reader may still run
            u.partials[2 * slot] = 0.0;
            u.partials[2 * slot + 1] = -1.0;
        }
        return;
    }
    sx_twiddles<V>(tw, twg);
    sx_rows<V>(sr, t, r0, t.a[1].w0, t.a[1].nw, t.a[2].w0, t.a[2].nw, g.P[1]);
    __syncthreads();
    pdl_wait();
    if ((g.clear & 2) && blockIdx.x + blockIdx.y + threadIdx.x == 0) bad_clear(g.bad, BAD_PSI);
    sx_flag(sr.flag, g.bad && epi != EPI_MUL_FIRST && epi != EPI_MUL_ACC ? &g.bad->any[BAD_QUOTIENT] : nullptr,
            [&] { sx_load_lines<V>(A, S + (long long)blockIdx.y * g.stride, (long long)g.Zs * g.P[1] * 16, sr.b); });
    __syncthreads();
    sx_p2<V, true>(A, tw);
    __syncthreads();
    float ksum = 0.0f, kcomp = 0.0f, kmax = -1.0f;
    const int x0 = t.a[0].w0, nx = t.a[0].nw;
    const unsigned long long pol = sep_policy(g.stream);
    const bool pairs = sx_pairs(vec, t.a[0], x0, nx);
    for (int it = threadIdx.x; it < SH::R * 16; it += SH::NT) {
        const int q = it & 15, row = it >> 4;
        const long long vb = sr.a[row];
        float2 *p = A + row * kSepRS + q;
        if constexpr (MUL) {
            float2 a[V];
#pragma unroll
            for (int k1 = 0; k1 < V; ++k1) a[k1] = p[k1 * SH::BS];
            sx_p1<V, true>(a, tw, q);
#pragma unroll
            for (int v = 0; v < V; ++v) p[v * SH::BS] = a[v];
        } else {
            if (vb < 0) continue;
            const int g0 = t.a[0].lo + 2 * q;
            if (pairs) sx_update_row<V, ST, true>(p, tw, q, u, vb, g0, x0, nx, ksum, kcomp, kmax, pol);
            else sx_update_row<V, ST, false>(p, tw, q, u, vb, g0, x0, nx, ksum, kcomp, kmax, pol);
        }
    }
    if constexpr (MUL) {
        __syncthreads();
        sx_mul_rows<V, ST>(A, u, epi, t, sr.a, ksum, kcomp, kmax, pol);
    }
    if (!ST && sr.flag) {
        __syncthreads();  // behind the rows' stores
#pragma unroll 1
        for (int i = threadIdx.x; i < SH::R * nx; i += SH::NT) {
            const int row = i / nx, x = x0 + i - row * nx, r = r0 + row;
            if (sr.a[row] >= 0 && bad_voxel(g.bad, x, t.a[1].w0 + r % t.a[1].nw, t.a[2].w0 + r / t.a[1].nw))
                sx_bad_value(u, MUL, sr.a[row] + x);
        }
    }
    if (ST) stats_to_partials(ksum, kcomp, kmax, red_s, red_m, u.partials, slot);
}

struct SxOps {
    int rows;  // per CTA
    cudaError_t (*ready)();  // on the current device, before the first launch there
    cudaError_t (*fwd)(const SepGeom &, const SepTiles &, int, int, const SepSrc &, float2 *, int, const float2 *,
                       cudaStream_t);
    cudaError_t (*ratio)(const SepGeom &, const SepTiles &, int, int, const float *, float2 *, int, const float2 *,
                         cudaStream_t, bool);
    cudaError_t (*update)(const SepGeom &, const SepTiles &, int, int, int, const SepUpd &, const float2 *, int,
                          const float2 *, cudaStream_t, bool);
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
        static PerDevice once;
        return once(limits);
    }
    static cudaError_t fwd(const SepGeom &g, const SepTiles &tl, int nt, int ctas, const SepSrc &src, float2 *S, int vec,
                           const float2 *tw, cudaStream_t s)
    {
        return launch_pdl(k_sep_x_fwd<V>, dim3(ctas, nt), SH::NT, SH::smem, s, src, S, tl, g, vec, tw);
    }
    static cudaError_t ratio(const SepGeom &g, const SepTiles &tl, int nt, int ctas, const float *img, float2 *S,
                             int vec, const float2 *tw, cudaStream_t s, bool first)
    {
        return launch_dep(first, k_sep_x_ratio<V>, dim3(ctas, nt), SH::NT, SH::smem, s, S, img, tl, g, vec, tw);
    }
    static cudaError_t update(const SepGeom &g, const SepTiles &tl, int nt, int ctas, int epi, const SepUpd &u,
                              const float2 *S, int vec, const float2 *tw, cudaStream_t s, bool first)
    {
        const dim3 grid(ctas, nt);
        const bool st = u.partials && (epi == EPI_SEQ || epi == EPI_MUL_FINAL);
#define SX_UPD(M, ST) launch_dep(first, k_sep_x_update<V, M, ST>, grid, SH::NT, SH::smem, s, S, u, epi, tl, g, vec, tw)
        if (epi == EPI_SEQ) return st ? SX_UPD(false, true) : SX_UPD(false, false);
        return st ? SX_UPD(true, true) : SX_UPD(true, false);
#undef SX_UPD
    }
    static const SxOps *ops()
    {
        static const SxOps o = {SH::R, &ready, &fwd, &ratio, &update};
        return &o;
    }
};

const SxOps *sx_ops_a(int n);
const SxOps *sx_ops_b(int n);
const SxOps *sx_ops_c(int n);

}  // namespace mvr
