// 3x3x3 convolution (stride 1, zero padding 1) on channels-last BF16 volumes as
// implicit GEMMs on the tcgen05 tensor cores, FP32 accumulation in tensor memory.
//
//   forward  Y[n][co] = act( sum_{t,ci} X[n + off(t)][ci] W[co][t][ci] + b[co] )
//   dgrad    dX[n][ci] = sum_{t,co} G[n - off(t)][co] W[co][t][ci]
//            the same kernel (conv3d_march.cuh) with the offsets negated and WT[ci][t][co] as B
//   wgrad    dW[co][t][ci] += sum_n G[n][co] X[n + off(t)][ci]
//            K = voxels, split over CTAs, FP32 atomics into dW
//
// Volumes are [B][D][H][W][C] (x fastest, then y, z, batch), C a multiple of 16.  Every wait is
// bounded and reports a timeout through err instead of hanging.
#pragma once
#include "tcgen05.cuh"

namespace mvr {

struct ConvGeom {
    int B, D, H, W;
    long long nvox;  // B * D * H * W
};

constexpr long long kTcWaitIter = 1LL << 24;

__device__ __forceinline__ void vox_coords(const ConvGeom &g, long long n, int &x, int &y, int &z, int &b)
{
    x = (int)(n % g.W);
    long long t = n / g.W;
    y = (int)(t % g.H);
    t /= g.H;
    z = (int)(t % g.D);
    b = (int)(t / g.D);
}

// 16-byte asynchronous copy global -> shared (L2 only); ok == false writes 16 zero bytes
// (source size 0, the source address not read)
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool ok)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(ok ? 16 : 0) : "memory");
}

}  // namespace mvr
