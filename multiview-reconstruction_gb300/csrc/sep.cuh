// Separable transforms on column blocks (sep_x.cuh, sep_yz.cuh): the FP32 convolutions of one
// iteration as row passes along x and tile passes along y and z, for FFT domains chosen by the
// library around a region of the volume (a "tile") instead of around the caller's block.
//
// Spectrum layout: 16 complex x columns (128 bytes) form a column block xb; a tile's spectrum is
// S[xb][z][y][16], so a y tile (one xb, one z) is one contiguous run and a z tile (one xb, one y)
// is one full line per z.  x has m = Px / 2 = 16 VX packed columns; column 0 carries X[0] +
// i X[m] along x and is split during the y pass, X[m]'s spectrum going to a plane of its own
// behind the blocks, N[z][y].  Frequencies stay in the order the two-phase transforms leave;
// K1^ and K2^ come from the same kernels, so the product is taken position by position.
//
// Along each axis a tile works on Px (Py, Pz) voxels from volume coordinate lo.  psi is needed on
// the written range plus twice the kernel's reach (only once beyond a face of the volume, where
// the quotient is the constant 1), the quotient on the written range plus once the reach.  Rows
// and planes that the mirror-single extension repeats are transformed along x once and read
// again by index; rows and planes outside the volume need no quotient at all: the spectrum of
// a constant row or plane is one known value.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace mvr {

// One axis of a tile.
struct SepAxis {
    int lo;      // volume coordinate of domain index 0
    int N;       // volume size
    int v0, nv;  // volume indices whose psi rows are transformed: [v0, v0 + nv)
    int q0, nq;  // volume indices whose quotient is formed
    int w0, nw;  // volume indices written
};
struct SepTile {
    SepAxis a[3];
};
constexpr int kSepMaxTiles = 16;
struct SepTiles {
    SepTile t[kSepMaxTiles];
};

// What every launch of a tile batch shares.
struct SepGeom {
    int P[3];          // FFT domain
    int nxb;           // column blocks, Px / 32
    int Zs;            // planes a tile's spectrum buffer holds
    long long stride;  // complex values per tile: nxb Zs Py 16 + Zs Py
    int stream;        // 1: volumes and K^ pass through L2 with the evict-first priority
    BadMap *bad;       // marks of the blocks that read values that are not finite (NULL: a block of its own)
    int clear;         // 1: the forward pass clears the quotients' marks, 2: the update psi's
};
inline SepGeom sep_geom(const int P[3], int planes)
{
    SepGeom g;
    for (int d = 0; d < 3; ++d) g.P[d] = P[d];
    g.nxb = P[0] / 32;
    g.Zs = planes;
    g.stride = ((long long)g.nxb * 16 + 1) * planes * P[1];
    g.stream = 0;
    g.bad = nullptr;
    g.clear = 0;
    return g;
}

// The column blocks [x0, x0 + n) of a y or z pass (the Nyquist plane goes with block 0).  first: the
// launch follows a join of streams (no programmatic dependence on its predecessor).
struct SepSlab {
    int x0, n;
    bool first;
};

// The smallest supported transform length >= n along x, and along y and z (0: none).
int sep_len_x(int n);
int sep_len_yz(int n);

struct SepSrc {
    const float *vol;  // psi volume (x, y, z sizes in the tiles), or a kernel of kd
    int kernel;        // 1: vol is a kernel, wrapped around the origin and scaled
    int kd[3];
    double scale;
};
struct SepUpd {
    const float *psi;     // source volume
    float *dst;           // output volume
    const float *img;     // the view's image (ratio pass)
    const float *weight[kMaxViews];
    int nviews;
    float2 *prod;         // running product over the views, volume layout
    UpdConst c;
    double *partials;     // {sum, max} per CTA, or NULL: no statistics
};

// Shared-memory opt-ins of the passes of a domain, on the current device: made with the plan, not asked for
// by each launch.
cudaError_t sep_ready(const int P[3]);

// x passes.  CTAs per tile of a pass over `rows` rows, and slots of its partials.
int sep_row_ctas(int Px, int rows);
cudaError_t sep_x_fwd(const SepGeom &g, const SepTiles &tl, int nt, const SepSrc &src, float2 *S, const float2 *twx,
                      cudaStream_t s);
cudaError_t sep_x_ratio(const SepGeom &g, const SepTiles &tl, int nt, const float *img, float2 *S, const float2 *twx,
                        cudaStream_t s, bool first = false);
// epi: EPI_SEQ, EPI_MUL_FIRST, EPI_MUL_ACC or EPI_MUL_FINAL
cudaError_t sep_x_update(const SepGeom &g, const SepTiles &tl, int nt, int epi, const SepUpd &u, const float2 *S,
                         const float2 *twx, cudaStream_t s, bool first = false);

// Where a pass finds its input rows or planes along the transformed axis.
enum SepMap {
    SEP_MIRROR = 0,  // psi: [v0, v0 + nv) under the mirror-single extension
    SEP_FILL = 1,    // quotient: [q0, q0 + nq), 1 elsewhere
    SEP_KERNEL = 2,  // kernel: taps wrapped around the origin, 0 elsewhere
};
// y passes in place, over planes [0, planes) of each tile's buffer: forward from the stored rows,
// inverse to the quotient's rows (out_w 0) or the written rows (out_w 1).
// kd: the kernel's size (SEP_KERNEL; else NULL).
cudaError_t sep_y_fwd(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, const int kd[3], float2 *S,
                      const float2 *twy, cudaStream_t s);
cudaError_t sep_y_inv(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int out_w, float2 *S, const float2 *twy,
                      cudaStream_t s);
// z pass: forward, times K, inverse; src planes by `map`, dst planes: the quotient's (out_w 0) or
// the written ones (out_w 1).  K NULL: forward alone, every plane of a kernel spectrum (dst with
// Zs = Pz) stored.
cudaError_t sep_z(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, int out_w, const int kd[3], const float2 *src,
                  float2 *dst, const float2 *K, const float2 *twz, cudaStream_t s);

}  // namespace mvr
