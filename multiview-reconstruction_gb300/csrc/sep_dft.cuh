// Register DFTs of the separable transforms (sep_x.cuh, sep_yz.cuh): lengths 2 ... 24 with
// compile-time twiddles.
#pragma once
#include "rows_warp.cuh"
#include "cols_tile.cuh"

namespace mvr {

// Global accesses with an L2 priority chosen at run time (SepGeom::stream): evict-first for what
// a pass reads or writes once, so that the spectrum that the next pass reads stays in L2.
__device__ __forceinline__ unsigned long long sep_policy(int stream)
{
    unsigned long long p;
    if (stream) asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    else asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Volumes are read with ordinary (coherent) loads: the update writes the volume it reads where psi is
// updated in place, and a kernel launched early runs beside the one that writes psi.  Volatile, so
// that the compiler keeps them behind pdl_wait.  6 views of 512 x 512 x 256 take 7.98 ms an iteration, as
// ld.global.nc 8.19; smaller volumes the same.
__device__ __forceinline__ float sep_ld(const float *p, unsigned long long pol)
{
    float v;
    asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ float2 sep_ld2(const void *p, unsigned long long pol)
{
    float2 v;
    asm volatile("ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(pol));
    return v;
}
// K^, which is never written while a pass runs.
__device__ __forceinline__ float2 sep_ldk(const void *p, unsigned long long pol)
{
    float2 v;
    asm("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ void sep_st(float *p, float v, unsigned long long pol)
{
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void sep_st2(void *p, float2 v, unsigned long long pol)
{
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(v.x), "f"(v.y), "l"(pol) : "memory");
}

// cos / sin of 2 pi j / n at compile time: the angle is reduced to the first octant by symmetry,
// then the Taylor series (in double; the constants are rounded to float where they are used).
struct SepCs {
    double c, s;
};
__host__ __device__ constexpr SepCs sep_cs(long long j, long long n)
{
    j %= n;
    if (j < 0) j += n;
    const long long o = 8 * j / n;  // octant
    // distance to the nearest multiple of a quarter turn, in units of 2 pi / (4 n)
    const long long quarter = (o + 1) / 2;
    const long long d4 = 4 * j - quarter * n;  // in [-n / 2, n / 2]
    const double x = 6.283185307179586476925286766559 * (double)d4 / (4.0 * (double)n);
    double c = 1.0, s = x, tc = 1.0, ts = x;
    for (int k = 1; k < 14; ++k) {
        tc *= -x * x / (double)((2 * k - 1) * (2 * k));
        ts *= -x * x / (double)((2 * k) * (2 * k + 1));
        c += tc;
        s += ts;
    }
    switch ((int)(quarter & 3)) {
    case 0: return SepCs{c, s};
    case 1: return SepCs{-s, c};
    case 2: return SepCs{-c, -s};
    default: return SepCs{s, -c};
    }
}

template <int N>
struct SepTab {
    float c[N], s[N];
};
template <int N>
__host__ __device__ constexpr SepTab<N> sep_tab()
{
    SepTab<N> t{};
    for (int j = 0; j < N; ++j) {
        const SepCs v = sep_cs(j, N);
        t.c[j] = (float)v.c;
        t.s[j] = (float)v.s;
    }
    return t;
}

// v times W_n^j = exp(-+2 pi i j / n) for a compile-time constant (c, s) = (cos, sin)(2 pi j / n)
template <bool INV>
__device__ __forceinline__ float2 sep_rot(float2 v, float c, float s)
{
    return INV ? make_float2(v.x * c - v.y * s, v.y * c + v.x * s) : make_float2(v.x * c + v.y * s, v.y * c - v.x * s);
}

// a + s b, both components with one fused paired instruction
__device__ __forceinline__ float2 sep_fma(float2 a, float2 b, float s)
{
#if MVR_PAIRED_FP && defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __ffma2_rn(b, make_float2(s, s), a);
#else
    return make_float2(fmaf(b.x, s, a.x), fmaf(b.y, s, a.y));
#endif
}
// (m - i n, m + i n) forward, the reverse inverse
template <bool INV>
__device__ __forceinline__ void sep_pm(float2 m, float2 n, float2 &p, float2 &q)
{
    p = make_float2(m.x + n.y, m.y - n.x);
    q = make_float2(m.x - n.y, m.y + n.x);
    if (INV) {
        const float2 t = p;
        p = q;
        q = t;
    }
}

// 5 points with fused products: 14 paired instructions and 8 additions
template <bool INV>
__device__ __forceinline__ void sep_dft5(float2 *v)
{
    constexpr SepTab<5> t = sep_tab<5>();
    const float2 a1 = cadd(v[1], v[4]), a2 = cadd(v[2], v[3]);
    const float2 b1 = csub(v[1], v[4]), b2 = csub(v[2], v[3]);
    const float2 m1 = sep_fma(sep_fma(v[0], a1, t.c[1]), a2, t.c[2]);
    const float2 m2 = sep_fma(sep_fma(v[0], a1, t.c[2]), a2, t.c[1]);
    const float2 n1 = sep_fma(cscale(b1, t.s[1]), b2, t.s[2]);
    const float2 n2 = sep_fma(cscale(b1, t.s[2]), b2, -t.s[1]);
    v[0] = cadd(v[0], cadd(a1, a2));
    sep_pm<INV>(m1, n1, v[1], v[4]);
    sep_pm<INV>(m2, n2, v[2], v[3]);
}

template <bool INV>
__device__ __forceinline__ void dft7(float2 *v)
{
    constexpr SepTab<7> t = sep_tab<7>();
    float2 a[3], b[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        a[q] = cadd(v[q + 1], v[6 - q]);
        b[q] = csub(v[q + 1], v[6 - q]);
    }
    const float2 v0 = v[0];
    v[0] = cadd(v0, cadd(a[0], cadd(a[1], a[2])));
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        float2 m = v0, n = cscale(b[0], t.s[k]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            m = sep_fma(m, a[q], t.c[((q + 1) * k) % 7]);
            if (q) n = sep_fma(n, b[q], t.s[((q + 1) * k) % 7]);
        }
        sep_pm<INV>(m, n, v[k], v[7 - k]);
    }
}

template <int N, bool INV>
__device__ __forceinline__ void sep_dft(float2 *v);

// N = A x B (Cooley-Tukey): inner A-point DFTs over q = B q1 + q2, twiddle W_N^(q2 k1), outer
// B-point DFTs; output k = k1 + A k2.
template <int A, int B, bool INV>
__device__ __forceinline__ void sep_ct(float2 *v)
{
    constexpr int N = A * B;
    constexpr SepTab<N> t = sep_tab<N>();
    float2 u[B][A];
#pragma unroll
    for (int q2 = 0; q2 < B; ++q2) {
#pragma unroll
        for (int q1 = 0; q1 < A; ++q1) u[q2][q1] = v[B * q1 + q2];
        sep_dft<A, INV>(u[q2]);
    }
#pragma unroll
    for (int q2 = 1; q2 < B; ++q2)
#pragma unroll
        for (int k1 = 1; k1 < A; ++k1) {
            const int j = q2 * k1;
            if (4 * j == N) u[q2][k1] = mul_j<INV>(u[q2][k1]);
            else if (2 * j == N) u[q2][k1] = make_float2(-u[q2][k1].x, -u[q2][k1].y);
            else u[q2][k1] = sep_rot<INV>(u[q2][k1], t.c[j], t.s[j]);
        }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        float2 w[B];
#pragma unroll
        for (int q2 = 0; q2 < B; ++q2) w[q2] = u[q2][k1];
        sep_dft<B, INV>(w);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = w[k2];
    }
}

template <int N, bool INV>
__device__ __forceinline__ void sep_dft(float2 *v)
{
    if constexpr (N == 2) dft2<INV>(v);
    else if constexpr (N == 3) dft3<INV>(v);
    else if constexpr (N == 4) dft4<INV>(v);
    else if constexpr (N == 5) sep_dft5<INV>(v);
    else if constexpr (N == 6) dft6<INV>(v);
    else if constexpr (N == 7) dft7<INV>(v);
    else if constexpr (N == 8) dft8<INV>(v);
    else if constexpr (N == 9) dft9<INV>(v);
    else if constexpr (N == 10) sep_ct<5, 2, INV>(v);
    else if constexpr (N == 12) dft12<INV>(v);
    else if constexpr (N == 14) sep_ct<7, 2, INV>(v);
    else if constexpr (N == 16) dft16<INV>(v);
    else if constexpr (N == 18) dft18<INV>(v);
    else if constexpr (N == 20) sep_ct<4, 5, INV>(v);
    else {
        static_assert(N == 24, "no register DFT of this length");
        sep_ct<8, 3, INV>(v);
    }
}

}  // namespace mvr
