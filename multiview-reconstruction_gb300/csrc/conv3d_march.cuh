// Forward and data-gradient 3x3x3 convolutions by columns of planes.
//
// A CTA walks a run of output planes, z fastest, of 8 x 16 columns of output voxels (x, y).  Every
// input plane of a column (10 x 18 voxels with its halo, zero outside the volume) is copied into shared
// memory once, through a ring of kMarchStages buffers, and multiplied once: the products of one offset
// (dy, dx) with the weights of all three dz give the plane's share of three output planes, so the
// three go into one product of 3 N columns whose accumulators are the tensor-memory columns of the
// output planes z - 1, z and z + 1.  These columns are a ring of R planes: an output plane is
// complete, and read back, once the input plane behind it has been multiplied.
//
// A K-group-major plane (the 16-byte chunk of channels 8j..8j+7 of halo voxel h = hx + 10 hy at byte
// j * kMarchLbo + 16 h) needs no copies per offset: eight x-consecutive voxels are one core matrix, the
// next line of the column is 10 rows further, and an offset is the same layout started
// 16 ((1 + dx) + 10 (1 + dy)) bytes later.
//
// What bounds it: the operands' way out of shared memory.  A product of 128 rows reads 4 KB of A however
// few columns it has, so 16 output channels at a time pay nine times for what 3 x 16 pay three times;
// with B's 1.5 KB a product of 48 columns took 48 cycles.  Taking dz into the columns
// divides the products by three (9 per 16 input channels and plane), loading a plane once divides
// the copies by three against bricks with a halo of three planes, and the weights (27 N C) come once
// per run instead of once per brick.  The products go out from one elected lane of a warp of its own:
// issued behind `threadIdx.x == 0`, with descriptors formed per product, the first layer below took
// 230 us, most of them one thread's chain of instructions.
// One layer on 128^3 voxels (64^3 for 96 channels), bricks before and runs after: 48 -> 16 channels
// 680 and 115 us, 16 -> 16 193 and 60, 96 -> 32 292 and 70; 16 -> 32 40 and 26, 32 -> 64 (32^3) 20 and 19.
#pragma once
#include "conv3d_tc.cuh"
#include "pdl.cuh"

namespace mvr {

constexpr int kMarchX = 8, kMarchY = 16;  // a column's lines: 128 rows of a product
constexpr int kMarchHX = kMarchX + 2, kMarchHY = kMarchY + 2, kMarchPlane = kMarchHX * kMarchHY;
constexpr int kMarchLbo = (kMarchPlane + 1) * 16;  // one padding row: distinct banks for the K groups
constexpr int kMarchStages = 4;
constexpr int kMarchThreads = 160;  // four warps copy planes and write results, one issues products

// Output channels of one CTA: all of them while the weights leave room for two CTAs or, with many
// input channels, for the ring of planes; the others are another CTA's, which reads the planes again.
template <int N, int C>
__host__ __device__ constexpr int march_ns()
{
    return N > 64 || 27 * N * C * 2 > 64 * 1024 ? N / 2 : N;
}
// tensor-memory columns of a CTA: a quarter of the SM's for the small channel counts, whose planes
// are short and need more CTAs in flight, else half
template <int NS, int C>
__host__ __device__ constexpr int march_cols()
{
    return NS <= 32 && C <= 16 ? 128 : 256;
}
template <int NS, int C>
__host__ __device__ constexpr size_t march_smem()
{
    return (size_t)kMarchStages * (C / 8) * kMarchLbo + 27 * (size_t)NS * C * 2 + 1024;
}

// A place in a CTA's run of output planes: the run goes through the planes of all columns, z fastest,
// and falls into parts of one column each.  A part of nz output planes has nz + 2 steps, one per input
// plane z = zs - 1 + p.
struct MarchAt {
    long long u;  // output plane of the run that the part starts at
    int x0, y0, zs, b, nz, p;
    __device__ __forceinline__ void start(const ConvGeom &g, long long u1)
    {
        const int nbx = (g.W + kMarchX - 1) / kMarchX, nby = (g.H + kMarchY - 1) / kMarchY;
        const long long col = u / g.D;
        zs = (int)(u - col * g.D);
        nz = (int)min((long long)(g.D - zs), u1 - u);
        x0 = (int)(col % nbx) * kMarchX;
        y0 = (int)(col / nbx % nby) * kMarchY;
        b = (int)(col / nbx / nby);
        p = 0;
    }
    // the next step; true at the start of a part
    __device__ __forceinline__ bool next(const ConvGeom &g, long long u1)
    {
        if (++p < nz + 2) return false;
        u += nz;
        if (u < u1) start(g, u1);
        return u < u1;
    }
};

// The copies of input planes, by 128 threads.  CU > 0: the input is the concatenation [nearest x2
// upsampling of `act` (CU channels, a volume of half the size), act2 (C - CU channels)].  kMarchHalf: `act`
// holds the lower half of the channels, the others are zero (a product takes 16, the network's input has two).
constexpr int kMarchHalf = -1;
template <int C, int CU>
struct MarchPlanes {
    static constexpr int CH = CU == kMarchHalf ? C / 16 : C / 8, ITEMS = kMarchPlane * CH, LI = (ITEMS + 127) / 128;
    static_assert(CU == kMarchHalf || (CU % 8 == 0 && CU >= 0 && CU < C), "concatenated channel split");
    const ConvGeom &g;
    const uint4 *act, *act2;
    int tid;
    // this thread's 16-byte chunks of a plane, channel chunk fastest: offset in chunks from the halo's
    // corner (x0 - 1, y0 - 1), of the low volume (x0 / 2 - 1, y0 / 2 - 1); -1 outside
    int off[LI];
    __device__ __forceinline__ MarchPlanes(const ConvGeom &g_, const __nv_bfloat16 *a, const __nv_bfloat16 *a2, int t)
        : g(g_), act(reinterpret_cast<const uint4 *>(a)), act2(reinterpret_cast<const uint4 *>(a2)), tid(t)
    {
    }
    __device__ __forceinline__ void column(const MarchAt &at)
    {
#pragma unroll
        for (int i = 0; i < LI; ++i) {
            const int k = tid + 128 * i, h = k / CH, j = k - h * CH;
            const int xx = at.x0 - 1 + h % kMarchHX, yy = at.y0 - 1 + h / kMarchHX;
            const bool in = k < ITEMS && xx >= 0 && yy >= 0 && xx < g.W && yy < g.H;
            if constexpr (CU <= 0) off[i] = in ? ((h / kMarchHX) * g.W + h % kMarchHX) * CH + j : -1;
            else if (j < CU / 8)
                off[i] = in ? ((h / kMarchHX + 1) / 2 * (g.W >> 1) + (h % kMarchHX + 1) / 2) * (CU / 8) + j : -1;
            else off[i] = in ? ((h / kMarchHX) * g.W + h % kMarchHX) * (CH - CU / 8) + j - CU / 8 : -1;
        }
    }
    // the K groups that are not stored, in every buffer, once
    __device__ __forceinline__ void clear(uint8_t *planes) const
    {
        if constexpr (CU == kMarchHalf)
            for (int k = tid; k < kMarchStages * CH * kMarchPlane; k += kMarchThreads) {
                const int g8 = k / kMarchPlane, st = g8 / CH;
                *reinterpret_cast<uint4 *>(planes + (st * 2 * CH + CH + g8 - st * CH) * kMarchLbo +
                                           16 * (k - g8 * kMarchPlane)) = make_uint4(0, 0, 0, 0);
            }
    }
    __device__ __forceinline__ void copy(const MarchAt &at, uint8_t *dst) const
    {
        auto corner = [&](int z, int D, int H, int W, int y, int x) {
            return (((long long)at.b * D + z) * H + y) * W + x;
        };
        const int z = at.zs - 1 + at.p;
        const bool zin = z >= 0 && z < g.D;
        const int zz = zin ? z : 0;
        const uint4 *lo, *hi = nullptr;
        if constexpr (CU <= 0) {
            lo = act + corner(zz, g.D, g.H, g.W, at.y0 - 1, at.x0 - 1) * CH;
        } else {
            lo = act + corner(zz >> 1, g.D >> 1, g.H >> 1, g.W >> 1, at.y0 / 2 - 1, at.x0 / 2 - 1) * (CU / 8);
            hi = act2 + corner(zz, g.D, g.H, g.W, at.y0 - 1, at.x0 - 1) * (CH - CU / 8);
        }
#pragma unroll
        for (int i = 0; i < LI; ++i) {
            const int k = tid + 128 * i, h = k / CH, j = k - h * CH;
            const bool in = zin && off[i] >= 0;
            const uint4 *src = CU <= 0 || j < CU / 8 ? lo : hi;
            if ((i + 1) * 128 <= ITEMS || k < ITEMS) cp_async16(dst + j * kMarchLbo + 16 * h, in ? src + off[i] : act, in);
        }
    }
};

// What becomes of the output.  The 2x2x2 sums and the head are formed from the accumulators: as kernels of
// their own they read everything back (16 channels on 128^3: averages 14 us and head 13 us, against 8
// and 5 more here; the 48-channel gradient on 4 x 64^3 written whole and summed after it 126 us, now 53).
enum MarchOut {
    MARCH_BF16,   // out: BF16 with bias (+ReLU when relu != 0); out2 (or NULL): its 2x2x2 averages, BF16
    MARCH_FP32,   // out: FP32, no bias
    MARCH_HEAD,   // out: FP32, one value per voxel: MARCH_BF16's 16 channels times wh, plus bh[0]
    MARCH_SPLIT,  // gradient of a concatenation: the first CB channels summed over 2x2x2 voxels into
                  // out, the others into out2, both FP32
};

// Sum of 16 channels over the four voxels (x, y) of a quad: lane bits 0 and 3.  Each lane keeps four
// channels, 8 (bit 0) + 4 (bit 3) onwards, and sends the others.
__device__ __forceinline__ void quad_sum(const float (&v)[16], float (&r)[4], int lane)
{
    const bool ox = lane & 1, oy = lane & 8;
    float h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = (ox ? v[j + 8] : v[j]) + __shfl_xor_sync(0xffffffffu, ox ? v[j] : v[j + 8], 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = (oy ? h[j + 4] : h[j]) + __shfl_xor_sync(0xffffffffu, oy ? h[j] : h[j + 4], 8);
}

template <int N, int C, int OUT, int CU = 0, int CB = 0>
__global__ void __launch_bounds__(kMarchThreads) k_conv3d_march(const __nv_bfloat16 *__restrict__ act,
                                                                const __nv_bfloat16 *__restrict__ wk,
                                                                const float *__restrict__ bias, void *out, ConvGeom g,
                                                                int sign, int relu, int *err,
                                                                const __nv_bfloat16 *__restrict__ act2, void *out2,
                                                                const float *__restrict__ wh,
                                                                const float *__restrict__ bh)
{
    constexpr int NS = march_ns<N, C>(), ST = kMarchStages, CH = C / 8;
    constexpr uint32_t COLS = march_cols<NS, C>();
    constexpr int R = (int)COLS / NS;  // ring of output planes: three being added to, one being read
    constexpr int PB = CH * kMarchLbo, B_TAP = 3 * NS * C * 2;
    static_assert(N % NS == 0 && NS % 16 == 0 && 3 * NS <= 256 && C % 16 == 0 && R >= 4, "tile shape");
    static_assert(OUT != MARCH_HEAD || NS == 16, "a thread holds the head's 16 channels");
    static_assert(CB % 16 == 0 && (OUT == MARCH_SPLIT) == (CB > 0), "channel split of the output");
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sB = smem + ((ST * PB + 1023) / 1024) * 1024;
    __shared__ __align__(8) uint64_t done[ST];
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (warp == 0) tc::tmem_alloc(&tbase, COLS);
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) tc::mbar_init(&done[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const long long planes =
        (long long)((g.W + kMarchX - 1) / kMarchX) * ((g.H + kMarchY - 1) / kMarchY) * g.B * g.D;
    const int pz = g.D & 1 ? 1 : 2;  // a run begins and ends between pairs of planes (sums over 2x2x2 voxels)
    const long long u1 = planes / pz * (blockIdx.x + 1) / gridDim.x * pz;
    const int co0 = blockIdx.y * NS;
    // the copies run kMarchStages - 1 steps ahead of the products, past the ends of parts
    MarchAt ld, at;
    ld.u = at.u = planes / pz * blockIdx.x / gridDim.x * pz;
    ld.start(g, u1);
    at.start(g, u1);
    MarchPlanes<C, CU> in(g, act, act2, tid);
    in.column(ld);
    in.clear(smem);
    auto load = [&](int s) {  // the next input plane, of step s, into its buffer
        in.copy(ld, smem + (s % ST) * PB);
        if (ld.next(g, u1)) in.column(ld);
    };
    // the weights, per offset (dy, dx) 3 NS rows: output plane z - 1 (dz = 1), z, z + 1, each NS channels
    for (int s = tid; s < 27 * NS * CH; s += kMarchThreads) {
        const int t = s / (3 * NS * CH), rem = s - t * (3 * NS * CH), r = rem / CH, j = rem - r * CH;
        const int i = r / NS, tz = (1 - i) * sign + 1;
        cp_async16(sB + t * B_TAP + tc::core_offset(r, 8 * j, C),
                   reinterpret_cast<const uint4 *>(
                       wk + ((long long)(co0 + r - i * NS) * 27 + 9 * tz + (sign > 0 ? t : 8 - t)) * C) + j, true);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // From here on this CTA has its tensor memory, so a next kernel that starts beside it (launch_pdl)
    // takes only what is left.  Every CTA of the kernel before has its own for the same reason, and the
    // weights above are older than that kernel.
    pdl_trigger();
    pdl_wait();
#pragma unroll 1
    for (int s = 0; s < ST; ++s) {
        if (ld.u < u1 && warp < 4) load(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, tbase, 0);
    const uint32_t hbase = tc::smem_u32(smem), bbase = tc::smem_u32(sB);
    int ring = 0;  // output planes of the parts before: plane j of a part has the columns of slot (ring + j) % R
    // the products of step s, issued by one lane; its share i goes to the part's output plane p - 2 + i
    auto products = [&](int s) {
        const int i0 = max(0, 2 - at.p), i1 = min(3, at.nz + 2 - at.p);  // the planes that the part has
        const int s0 = (ring + at.p - 2 + i0) % R;                      // ring slot of the first
        const int n0 = min(i1 - i0, R - s0), n1 = i1 - i0 - n0;          // columns up to the ring's end, and from its start
        const uint64_t a0 = tc::smem_desc(hbase + (uint32_t)(s % ST) * PB, kMarchLbo, kMarchHX * 16);
        const uint64_t b0 = tc::smem_desc(bbase, 128, C * 16);
        // the newest output plane starts here, the others go on
        for (int i = i0; i < i1; ++i)
            tc::mma_bf16(tmem + (uint32_t)((ring + at.p - 2 + i) % R * NS), a0, b0 + (uint32_t)(i * NS * C * 2 / 16),
                         tc::idesc_bf16(128, NS), i != 2);
#pragma unroll 1
        for (int seg = 0; seg < (n1 > 0 ? 2 : 1); ++seg) {
            const int n = seg ? n1 : n0, i = seg ? i0 + n0 : i0;
            const uint32_t d = tmem + (seg ? 0u : (uint32_t)(s0 * NS));
            const uint32_t id = tc::idesc_bf16(128, NS) + ((uint32_t)((n - 1) * (NS >> 3)) << 17);
            const uint64_t bs = b0 + (uint32_t)(i * NS * C * 2 / 16);
#pragma unroll
            for (int t = 0; t < 9; ++t)
#pragma unroll
                for (int k = 0; k < C / 16; ++k)
                    if (t > 0 || k > 0)
                        tc::mma_bf16_acc(d, a0 + (uint32_t)(2 * k * kMarchLbo / 16 + t % 3 + kMarchHX * (t / 3)),
                                         bs + (uint32_t)(t * B_TAP / 16 + k * 16), id);
        }
        tc::mma_commit(&done[s % ST]);
    };
    bool ok = true;
    int s = 0, slot = -1;  // slot of the output plane that step s - 1 completed, or -1
    long long n = 0;       // this thread's voxel of it, and the voxel of the half-size volume
    long long nl = 0;
    bool rv = false, odd = false;
    const int lane = tid & 31;
    const bool pool = OUT == MARCH_BF16 && out2 != nullptr;
    float pair[NS / 16][4];  // the quad's sums of an even plane
#pragma unroll 1
    for (;; ++s) {
        const bool more = at.u < u1;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");  // step s's plane has landed
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;  // the whole CTA
        if (more && warp == 4) {
            tc::fence_after_sync();
            if (tc::elect_one()) products(s);
            __syncwarp();
        }
        if (s > 0 && warp < 4) {
            // while step s is multiplied: step s - 1's buffer is free and its output plane complete
            ok = __all_sync(0xffffffffu, tc::mbar_wait(&done[(s - 1) % ST], ((s - 1) / ST) & 1, kTcWaitIter));
            if (ok && ld.u < u1) load(s - 1 + ST);  // on a timeout this warp writes no more
            tc::fence_after_sync();
            if (ok && slot >= 0) {
                const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(slot * NS);
#pragma unroll
                for (int c0 = 0; c0 < NS; c0 += 16) {
                    float v[16];
                    tc::tmem_ld16(trow + c0, v);
                    if constexpr (OUT == MARCH_BF16 || OUT == MARCH_HEAD) {
                        __align__(16) __nv_bfloat16 w[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            float a = v[j] + (bias ? bias[co0 + c0 + j] : 0.0f);
                            if (relu) a = fmaxf(a, 0.0f);
                            w[j] = __float2bfloat16(a);
                            v[j] = __bfloat162float(w[j]);
                        }
                        if constexpr (OUT == MARCH_HEAD) {
                            float h = bh[0];
#pragma unroll
                            for (int j = 0; j < 16; ++j) h += wh[j] * v[j];
                            if (rv) static_cast<float *>(out)[n] = h;
                        } else if (rv) {
                            uint4 *op = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(out) + n * N + co0 + c0);
                            op[0] = reinterpret_cast<const uint4 *>(w)[0];
                            op[1] = reinterpret_cast<const uint4 *>(w)[1];
                        }
                    }
                    if ((OUT == MARCH_SPLIT && co0 + c0 < CB) || (OUT == MARCH_BF16 && pool)) {
                        float (&q)[4] = pair[c0 / 16];
                        float r[4];
                        quad_sum(v, r, lane);
                        if (!odd) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) q[j] = r[j];
                        } else if (rv) {
                            const int c = co0 + c0 + (lane & 1) * 8 + (lane >> 3 & 1) * 4;
                            if constexpr (OUT == MARCH_SPLIT) {
                                *reinterpret_cast<float4 *>(static_cast<float *>(out) + nl * CB + c) =
                                    make_float4(q[0] + r[0], q[1] + r[1], q[2] + r[2], q[3] + r[3]);
                            } else {
                                __align__(8) __nv_bfloat16 w[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j) w[j] = __float2bfloat16(0.125f * (q[j] + r[j]));
                                *reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(out2) + nl * N + c) =
                                    *reinterpret_cast<const uint2 *>(w);
                            }
                        }
                    } else if ((OUT == MARCH_SPLIT || OUT == MARCH_FP32) && rv) {
                        float4 *op = reinterpret_cast<float4 *>(
                            OUT == MARCH_SPLIT ? static_cast<float *>(out2) + n * (N - CB) + co0 + c0 - CB
                                               : static_cast<float *>(out) + n * N + co0 + c0);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            op[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (!more) break;
        slot = -1;
        if (at.p >= 2) {
            const int x = at.x0 + (tid & 7), y = at.y0 + (tid >> 3 & 15);
            slot = (ring + at.p - 2) % R;
            const int z = at.zs + at.p - 2;
            n = (((long long)at.b * g.D + z) * g.H + y) * g.W + x;
            nl = (((long long)at.b * (g.D >> 1) + (z >> 1)) * (g.H >> 1) + (y >> 1)) * (g.W >> 1) + (x >> 1);
            odd = z & 1;
            rv = x < g.W && y < g.H;
        }
        const int nz = at.nz;
        if (at.next(g, u1)) ring = (ring + nz) % R;
    }
    if (!__syncthreads_and(ok)) {
        // a wait ran out: let every copy and product in flight finish (bounded) before the tensor
        // memory goes back
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (tid == 0) {
            atomicExch(err, 1);
            for (int q = max(0, s - ST); q < s; ++q) tc::mbar_wait(&done[q % ST], (q / ST) & 1, kTcWaitIter);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, COLS);
}

// Weight gradient over the same runs: dW[co][t][ci] += sum_n G[n][co] X[n + off(t)][ci].
//
// The contraction runs over voxels: both operands are M/N-major, the 8 channels (16 bytes) of one voxel
// one core matrix row and 8 x-consecutive voxels one core matrix, so a plane of X in shared memory is
// the A operand of every offset (dy, dx) by its start address alone, and three consecutive planes
// of G in their ring are B for the three dz: product columns (i, co) of the offset's accumulators, G
// plane z - 1 + i against X plane z.  The accumulators of all offsets stay in tensor memory
// through the run (3 N columns each; with more output channels a CTA takes part of the offsets) and
// go into dW with FP32 atomics at its end.  Rows beyond C are read from whatever follows the
// plane and dropped.
//
// What bounds it: the operands' way out of shared memory, 2 KB of A (64 rows; 4 KB for more than 64
// channels) and 1.5 KB of B per product.  48 x 16 channels on
// 4 x 64^3 voxels: 97 us (0.85 ms with 27 copies of X out of L2, one per offset), 16 x 16, 8 of them stored: 34 us
// (0.30), 96 x 32 on 4 x 32^3: 42 us (0.25), 16 x 32: 21 us (0.048).  A column's ragged edge multiplies G's zeros with the X beside
// it: an X that is not finite reaches the outward offsets there, and what is not finite at the end of a run with
// ragged columns is summed again without the tensor cores (wgrad_again).
constexpr int kWgRing = 8;  // planes of G: three being multiplied, the others on their way
constexpr int kWgGroup = 128 * 16 + 16;  // stride of G's channel groups (padding: distinct banks)
// Up to 16 channels the 64 rows of a product are eight x shifts of one channel group, 16 bytes apart, of which
// the first three are dx = -1, 0, 1: a product per (dy, channel group) instead of one per (dy, dx) (16 x 16: 95 -> 44 us).
template <int C, int CU>
__host__ __device__ constexpr int wgrad_units()  // products of one K step
{
    return C > 16 ? 9 : 3 * (CU == kMarchHalf ? C / 16 : C / 8);
}
template <int N, int C, int CU>
__host__ __device__ constexpr int wgrad_splits()  // CTAs that share them: 512 columns hold 512 / (3 N)
{
    return (wgrad_units<C, CU>() + 512 / (3 * N) - 1) / (512 / (3 * N));
}
// tensor-memory columns of a CTA (a power of two); with few of them two CTAs share an SM (16 x 16: 44 -> 34 us)
template <int N, int C, int CU>
__host__ __device__ constexpr int wgrad_cols()
{
    constexpr int S = wgrad_splits<N, C, CU>(), n = (wgrad_units<C, CU>() + S - 1) / S * 3 * N;
    return n <= 128 ? 128 : (n <= 256 ? 256 : 512);
}
template <int N, int C>
__host__ __device__ constexpr size_t wgrad_march_smem()
{
    return (size_t)kMarchStages * (C / 8) * kMarchLbo + (size_t)kWgRing * (N / 8) * kWgGroup;
}

// Element (tap, ci, co) of the run's share, plain sums over the voxels of the volume.
template <int N, int C, int CU>
__device__ __forceinline__ float wgrad_again(const __nv_bfloat16 *X, const __nv_bfloat16 *X2, const __nv_bfloat16 *G,
                                             const ConvGeom &g, long long u0, long long u1, int tap, int ci, int co)
{
    const int dz = tap / 9 - 1, dy = tap / 3 % 3 - 1, dx = tap % 3 - 1;
    float s = 0.0f;
    MarchAt at;
#pragma unroll 1
    for (long long u = u0; u < u1; ++u) {
        at.u = u;
        at.start(g, u1);
        const int z = at.zs + dz;
        if (z < 0 || z >= g.D) continue;
#pragma unroll 1
        for (int v = 0; v < 128; ++v) {
            const int x = at.x0 + (v & 7), y = at.y0 + (v >> 3), xx = x + dx, yy = y + dy;
            if (x >= g.W || y >= g.H || xx < 0 || yy < 0 || xx >= g.W || yy >= g.H) continue;
            const long long n = (((long long)at.b * g.D + z) * g.H + yy) * g.W + xx;
            __nv_bfloat16 a;
            if constexpr (CU == kMarchHalf) a = ci < C / 2 ? X[n * (C / 2) + ci] : __float2bfloat16(0.0f);
            else if constexpr (CU == 0) a = X[n * C + ci];
            else if (ci >= CU) a = X2[n * (C - CU) + ci - CU];
            else
                a = X[((((long long)at.b * (g.D >> 1) + (z >> 1)) * (g.H >> 1) + (yy >> 1)) * (g.W >> 1) + (xx >> 1)) * CU + ci];
            s += __bfloat162float(G[((((long long)at.b * g.D + at.zs) * g.H + y) * g.W + x) * N + co]) * __bfloat162float(a);
        }
    }
    return s;
}

// RAGGED: a kernel of its own, whose registers cost the other 1 to 5 %.  One check per 16 sums, behind which they are
// added as without it: a training step on 60 x 36 x 40 takes 347 us, 339 unchecked, 558 with every sum picked out and checked.
template <int N, int C, int CU, bool RAGGED>
__global__ void __launch_bounds__(kMarchThreads) k_wgrad_march(const __nv_bfloat16 *__restrict__ X,
                                                               const __nv_bfloat16 *__restrict__ G, float *dW,
                                                               ConvGeom g, int *err,
                                                               const __nv_bfloat16 *__restrict__ X2 = nullptr)
{
    constexpr int ST = kMarchStages, RG = kWgRing, CH = C / 8, PB = CH * kMarchLbo, GB = (N / 8) * kWgGroup;
    constexpr int M = C <= 64 ? 64 : 128;
    constexpr bool XS = C <= 16;  // x shifts in the rows
    constexpr uint32_t COLS = wgrad_cols<N, C, CU>();
    constexpr int NU = wgrad_units<C, CU>(), NJ = XS ? NU / 3 : 1;
    static_assert(C <= 128 && N % 16 == 0 && 3 * N <= 256, "tile shape");
    // A's rows beyond C end inside the ring of G
    static_assert((M / 8 - CH) * kMarchLbo <= RG * GB, "rows beyond C stay in shared memory");
    static_assert(ST + 2 <= RG, "a plane of G is copied when its slot's last products are done");
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sG = smem + ST * PB;
    __shared__ __align__(8) uint64_t done[ST];
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (warp == 0) tc::tmem_alloc(&tbase, COLS);
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) tc::mbar_init(&done[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const long long planes =
        (long long)((g.W + kMarchX - 1) / kMarchX) * ((g.H + kMarchY - 1) / kMarchY) * g.B * g.D;
    const long long u1 = planes * (blockIdx.x + 1) / gridDim.x;
    const int t0 = NU * blockIdx.y / gridDim.y, t1 = NU * (blockIdx.y + 1) / gridDim.y;
    MarchAt ld, at;
    ld.u = at.u = planes * blockIdx.x / gridDim.x;
    ld.start(g, u1);
    at.start(g, u1);
    MarchPlanes<C, CU> in(g, X, X2, tid);
    in.column(ld);
    int lring = 0;  // output planes of the parts before: plane j of a part is in slot (ring + j) % RG
    auto load = [&](int s) {  // the next plane of X, of step s, and of G
        in.copy(ld, smem + (s % ST) * PB);
        if (ld.p < ld.nz) {
            uint8_t *dst = sG + (lring + ld.p) % RG * GB;
            const long long z = (long long)ld.b * g.D + ld.zs + ld.p;
#pragma unroll
            for (int i = 0; i < N / 8; ++i) {
                const int k = tid + 128 * i, v = k / (N / 8), j = k - v * (N / 8);
                const int x = ld.x0 + (v & 7), y = ld.y0 + (v >> 3);
                const bool ok = x < g.W && y < g.H;
                cp_async16(dst + j * kWgGroup + 16 * v, ok ? G + ((z * g.H + y) * g.W + x) * N + 8 * j : G, ok);
            }
        }
        const int nz = ld.nz;
        if (ld.next(g, u1)) {
            lring = (lring + nz) % RG;
            in.column(ld);
        }
    };
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    pdl_trigger();  // behind the allocation, as above
    pdl_wait();
#pragma unroll 1
    for (int s = 0; s < ST; ++s) {
        if (ld.u < u1 && warp < 4) load(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, tbase, 0);
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    if (warp < 4)
        for (int c = 0; c < (t1 - t0) * 3 * N; c += 16) tc::tmem_zero16(trow + c);
    const uint32_t xbase = tc::smem_u32(smem), gbase = tc::smem_u32(sG);
    int ring = 0;
    auto products = [&](int s) {  // issued by one lane
        const int i0 = max(0, 2 - at.p), i1 = min(3, at.nz + 2 - at.p);
        const int s0 = (ring + at.p - 2 + i0) % RG;
        const int n0 = min(i1 - i0, RG - s0), n1 = i1 - i0 - n0;  // planes up to the ring's end, and from its start
        const uint64_t a0 = tc::smem_desc(xbase + (uint32_t)(s % ST) * PB, kMarchHX * 16, XS ? 16 : kMarchLbo);
        const uint64_t b0 = tc::smem_desc(gbase, 128, kWgGroup);
#pragma unroll 1
        for (int seg = 0; seg < (n1 > 0 ? 2 : 1); ++seg) {
            const int n = seg ? n1 : n0, i = seg ? i0 + n0 : i0;
            const uint32_t id = tc::idesc_bf16_mn(M, N) + ((uint32_t)((n - 1) * (N >> 3)) << 17);
            const uint64_t bs = b0 + (seg ? 0u : (uint32_t)(s0 * (GB / 16)));
            uint32_t d = tmem + (uint32_t)(i * N);
#pragma unroll 1
            for (int t = t0; t < t1; ++t, d += 3 * N) {
                const uint64_t as = a0 + (uint32_t)(XS ? kMarchHX * (t / NJ) + t % NJ * (kMarchLbo / 16) : t % 3 + kMarchHX * (t / 3));
#pragma unroll
                for (int k = 0; k < 8; ++k) tc::mma_bf16_acc(d, as + 2 * kMarchHX * k, bs + 16 * k, id);
            }
        }
        tc::mma_commit(&done[s % ST]);
    };
    bool ok = true;
    int s = 0;
#pragma unroll 1
    for (;; ++s) {
        const bool more = at.u < u1;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");  // step s's planes have landed
        tc::fence_proxy_async();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;  // the whole CTA
        if (more && warp == 4) {
            tc::fence_after_sync();
            if (tc::elect_one()) products(s);
            __syncwarp();
        }
        if (s > 0 && warp < 4) {
            ok = __all_sync(0xffffffffu, tc::mbar_wait(&done[(s - 1) % ST], ((s - 1) / ST) & 1, kTcWaitIter));
            if (ok && ld.u < u1) load(s - 1 + ST);  // on a timeout this warp writes no more
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (!more) break;
        const int nz = at.nz;
        if (at.next(g, u1)) ring = (ring + nz) % RG;
    }
    tc::fence_after_sync();
    if (!__syncthreads_and(ok)) {
        // a wait ran out: let every copy and product in flight finish (bounded) before the tensor
        // memory goes back
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (tid == 0) {
            atomicExch(err, 1);
            for (int q = max(0, s - ST); q < s; ++q) tc::mbar_wait(&done[q % ST], (q / ST) & 1, kTcWaitIter);
        }
    } else if (warp < 4) {
        // row r is lane r, of 64 rows lanes 0..15 of each warp; every CTA starts at an offset of its own
        const int r = M == 64 ? 16 * warp + lane : 32 * warp + lane;
        const bool rv = r < (XS ? 24 : C) && (M == 128 || lane < 16);
        const int nt = t1 - t0;
#pragma unroll 1
        for (int q = 0; q < nt * 3; ++q) {
            const int e = (q + (int)blockIdx.x) % (nt * 3), t = t0 + e / 3, tz = 2 - e % 3;
            const int ci = XS ? 8 * (t % NJ) + r % 8 : r, tap = 9 * tz + (XS ? 3 * (t / NJ) + r / 8 : t);
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 16) {
                float v[16];
                tc::tmem_ld16(trow + (uint32_t)(e * N + c0), v);
                bool finite = true;
                if constexpr (RAGGED)
#pragma unroll
                    for (int j = 0; j < 16; ++j) finite = finite && fabsf(v[j]) <= 3.402823466e38f;
                if (rv && finite)
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        atomicAdd(&dW[((long long)(c0 + j) * 27 + tap) * C + ci], v[j]);
                if constexpr (RAGGED) {
                    if (rv && !finite)
#pragma unroll 1
                        for (int j = 0; j < 16; ++j) {
                            float a = v[0];
#pragma unroll
                            for (int i = 1; i < 16; ++i) a = i == j ? v[i] : a;
                            if (!(fabsf(a) <= 3.402823466e38f))
                                a = wgrad_again<N, C, CU>(X, X2, G, g, planes * blockIdx.x / gridDim.x, u1, tap, ci, c0 + j);
                            atomicAdd(&dW[((long long)(c0 + j) * 27 + tap) * C + ci], a);
                        }
                    __syncwarp();
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, COLS);
}

}  // namespace mvr
