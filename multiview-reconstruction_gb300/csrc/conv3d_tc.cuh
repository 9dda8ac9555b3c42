// 3x3x3 convolution (stride 1, zero padding 1) on channels-last BF16 volumes as
// implicit GEMMs on the tcgen05 tensor cores, FP32 accumulation in tensor memory.
//
//   forward  Y[n][co] = act( sum_{t,ci} X[n + off(t)][ci] W[co][t][ci] + b[co] )
//   dgrad    dX[n][ci] = sum_{t,co} G[n - off(t)][co] W[co][t][ci]
//            the same kernel (conv3d_march.cuh) with the offsets negated and WT[ci][t][co] as B
//   wgrad    dW[co][t][ci] += sum_n G[n][co] X[n + off(t)][ci]
//            M = 128 (t, ci) rows per CTA, N = C_out, K = voxels (split over CTAs,
//            FP32 atomics into dW)
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
template <int N>
struct TmemCols {
    static constexpr uint32_t value = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
};

// wgrad: D[(t,ci) rows][co] over the voxels [blockIdx.y * vpc, +vpc), atomically added
// to dW[co][t][ci] (FP32).
//
// The contraction runs over voxels and the activations are channels-last, so both operands are
// staged M/N-major: the 8 channels (16 bytes) of one voxel and tap are one core matrix row, and a
// stage is filled by 16-byte asynchronous copies alone, kWgStages - 2 stages ahead of the
// products (K-major staging transposed every channel group with eight 2-byte stores and formed the
// voxel's coordinates once per group: 16 x 48 channels on 4 x 64^3 voxels 1.93 ms).  A thread keeps
// one voxel of the stage and 8 row groups, whose taps are fixed for the whole kernel.
constexpr int kWgStages = 4;
constexpr int kWgKT = 64;  // voxels per stage
template <int N>
__host__ __device__ constexpr int wgrad_stage_bytes()
{
    return (128 + N) * kWgKT * 2;
}

template <int N, int C>
__global__ void __launch_bounds__(128) k_wgrad_tc(const __nv_bfloat16 *__restrict__ X,
                                                  const __nv_bfloat16 *__restrict__ G, float *dW, ConvGeom g,
                                                  long long vpc, int *err)
{
    constexpr int KT = kWgKT, ST = kWgStages;
    constexpr int A_BYTES = 128 * KT * 2, S_BYTES = wgrad_stage_bytes<N>();
    constexpr int ROWS = 27 * C;
    constexpr int BG = (N / 8) * KT / 128;  // channel groups of G per thread
    static_assert(BG * 128 == (N / 8) * KT, "whole rounds");
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar[ST];
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t ncols = TmemCols<N>::value;
    if (warp == 0) tc::tmem_alloc(&tbase, ncols);
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) tc::mbar_init(&mbar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tbase;
    const int row0 = blockIdx.x * 128;
    const long long n0 = (long long)blockIdx.y * vpc;
    const long long n1 = n0 + vpc < g.nvox ? n0 + vpc : g.nvox;
    const int stages = n1 > n0 ? (int)((n1 - n0 + KT - 1) / KT) : 0;
    const uint32_t idesc = tc::idesc_bf16_mn(128, N);
    // this thread's voxel of a stage and its row groups rg0 + 2 i: tap offsets in elements, and the tap
    const int k = tid & (KT - 1), rg0 = tid >> 6;
    long long toff[8];
    int tap[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = row0 + 8 * (rg0 + 2 * i), t = r / C;
        const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
        toff[i] = (((long long)dz * g.H + dy) * g.W + dx) * C + r % C;
        tap[i] = r < ROWS ? (dx + 1) | (dy + 1) << 2 | (dz + 1) << 4 : -1;
    }
    auto issue = [&](int s) {
        uint8_t *sa = smem + (s % ST) * S_BYTES, *sb = sa + A_BYTES;
        const long long nn = n0 + (long long)s * KT + k;
        const bool in = nn < n1;
        int x = 0, y = 0, z = 0, b = 0;
        if (in) {
            if (g.nvox <= 0x7fffffffLL) {
                const unsigned q = (unsigned)nn, t = q / (unsigned)g.W, u = t / (unsigned)g.H;
                x = (int)(q - t * g.W);
                y = (int)(t - u * g.H);
                z = (int)(u % (unsigned)g.D);
            } else {
                vox_coords(g, nn, x, y, z, b);
            }
        }
        // bit d set: the neighbour at offset d - 1 lies inside
        const int mx = (x > 0 ? 1 : 0) | 2 | (x + 1 < g.W ? 4 : 0), my = (y > 0 ? 1 : 0) | 2 | (y + 1 < g.H ? 4 : 0),
                  mz = (z > 0 ? 1 : 0) | 2 | (z + 1 < g.D ? 4 : 0);
        const __nv_bfloat16 *xp = X + nn * C;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool ok = in && tap[i] >= 0 && (mx >> (tap[i] & 3) & my >> (tap[i] >> 2 & 3) & mz >> (tap[i] >> 4) & 1);
            cp_async16(sa + (rg0 + 2 * i) * (KT * 16) + k * 16, ok ? xp + toff[i] : X, ok);
        }
#pragma unroll
        for (int i = 0; i < BG; ++i) {
            const int cg = rg0 + 2 * i;
            cp_async16(sb + cg * (KT * 16) + k * 16, in ? G + nn * N + 8 * cg : G, in);
        }
    };
    bool ok = true;
    int done = 0;  // stages whose products were issued
#pragma unroll 1
    for (int s = 0; s < ST - 2; ++s) {
        if (s < stages) issue(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
#pragma unroll 1
    for (int s = 0; s < stages; ++s) {
        const int nx = s + ST - 2;
        if (nx < stages) {
            // the buffer's last products (stage nx - ST); on a timeout this thread writes no more
            if (nx >= ST) ok = tc::mbar_wait(&mbar[nx % ST], ((nx - ST) / ST) & 1, kTcWaitIter);
            if (ok) issue(nx);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");  // stage s has landed
        tc::fence_proxy_async();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;  // the whole CTA
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t sa = tc::smem_u32(smem + (s % ST) * S_BYTES);
#pragma unroll
            for (int c = 0; c < KT / 16; ++c) {
                const uint64_t ad = tc::smem_desc(sa + c * 256, 128, KT * 16);
                const uint64_t bd = tc::smem_desc(sa + A_BYTES + c * 256, 128, KT * 16);
                tc::mma_bf16(tmem, ad, bd, idesc, (s > 0 || c > 0) ? 1 : 0);
            }
            tc::mma_commit(&mbar[s % ST]);
        }
        ++done;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    for (int s = max(0, done - ST); s < done; ++s) ok = tc::mbar_wait(&mbar[s % ST], (s / ST) & 1, kTcWaitIter) && ok;
    tc::fence_after_sync();
    ok = __syncthreads_and(ok) != 0;  // one outcome for the whole CTA (the TMEM loads are warp-wide)
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
    } else if (stages > 0) {
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        const int r = row0 + tid;  // (t, ci)
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tc::tmem_ld16(trow + c0, v);
            if (r < ROWS)
#pragma unroll
                for (int j = 0; j < 16; ++j) atomicAdd(&dW[(long long)(c0 + j) * ROWS + r], v[j]);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

}  // namespace mvr
