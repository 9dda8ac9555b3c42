// Register DFTs of the separable transforms (sep_x.cuh, sep_yz.cuh): lengths 2 ... 24 with
// compile-time twiddles.
#pragma once
#include "rows_warp.cuh"
#include "cols_tile.cuh"

namespace mvr {

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
        float2 m = v0, n = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float c = t.c[((q + 1) * k) % 7], s = t.s[((q + 1) * k) % 7];
            m = make_float2(fmaf(a[q].x, c, m.x), fmaf(a[q].y, c, m.y));
            n = make_float2(fmaf(b[q].x, s, n.x), fmaf(b[q].y, s, n.y));
        }
        // forward m - i n, inverse m + i n
        if (INV) {
            v[k] = make_float2(m.x - n.y, m.y + n.x);
            v[7 - k] = make_float2(m.x + n.y, m.y - n.x);
        } else {
            v[k] = make_float2(m.x + n.y, m.y - n.x);
            v[7 - k] = make_float2(m.x - n.y, m.y + n.x);
        }
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
    else if constexpr (N == 5) dft5<INV>(v);
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
