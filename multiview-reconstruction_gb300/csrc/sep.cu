// Host side of the separable transforms (see sep.cuh): lengths and launches.
#include "sep.cuh"

#include "sep_x.cuh"
#include "sep_yz.cuh"

#include <algorithm>
#include <cstdint>

namespace mvr {

namespace {

// Lengths with compiled passes.  x: 32 V (V-point DFTs, 16 packed columns per block).  y and z:
// T V with T and V register DFTs of 4 ... 24 points.  A size one above a length pads most: 50 % at 33 (y, z)
// and 65 (x), 20 % at 161, 321 (x) and 481 (y, z), 13 to 17 % elsewhere above 128.  Even so a block there is faster than
// its plan, whose domain hardly pads: 33 x 33 rows of 65 voxels 29 against 73 us, 161^3 100 / 289, 321^3 659 / 1700,
// 481^3 2.18 / 7.86 ms.
constexpr int kLenX[] = {64, 96, 128, 160, 192, 224, 256, 288, 320, 384, 448, 512, 576};
constexpr int kLenYZ[] = {32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 256, 288, 320, 360, 400, 432, 480, 576};

const SxOps *sx_ops(int n)
{
    const SxOps *o = sx_ops_a(n);
    if (!o) o = sx_ops_b(n);
    if (!o) o = sx_ops_c(n);
    return o;
}
const YzOps *yz_ops(int n)
{
    const YzOps *o = yz_ops_a(n);
    if (!o) o = yz_ops_b(n);
    if (!o) o = yz_ops_c(n);
    if (!o) o = yz_ops_d(n);
    return o;
}

template <class F>
int tile_max(const SepTiles &tl, int nt, F f)
{
    int m = 0;
    for (int i = 0; i < nt; ++i) m = std::max(m, f(tl.t[i]));
    return m;
}

bool aligned8(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }

}  // namespace

int sep_len_x(int n)
{
    for (int l : kLenX)
        if (l >= n) return l;
    return 0;
}
int sep_len_yz(int n)
{
    for (int l : kLenYZ)
        if (l >= n) return l;
    return 0;
}

int sep_row_ctas(int Px, int rows)
{
    const SxOps *o = sx_ops(Px);
    return o ? (rows + o->rows - 1) / o->rows : 0;
}

cudaError_t sep_ready(const int P[3])
{
    const SxOps *x = sx_ops(P[0]);
    const YzOps *y = yz_ops(P[1]), *z = yz_ops(P[2]);
    if (!x || !y || !z) return cudaErrorInvalidValue;
    cudaError_t e = x->ready();
    if (e == cudaSuccess) e = y->ready();
    return e == cudaSuccess ? z->ready() : e;
}

cudaError_t sep_x_fwd(const SepGeom &g, const SepTiles &tl, int nt, const SepSrc &src, float2 *S, const float2 *twx,
                      cudaStream_t s)
{
    const SxOps *o = sx_ops(g.P[0]);
    if (!o) return cudaErrorInvalidValue;
    const int rows = src.kernel ? src.kd[1] * src.kd[2]
                                : tile_max(tl, nt, [](const SepTile &t) { return t.a[1].nv * t.a[2].nv; });
    return o->fwd(g, tl, nt, sep_row_ctas(g.P[0], rows), src, S, aligned8(src.vol), twx, s);
}

cudaError_t sep_x_ratio(const SepGeom &g, const SepTiles &tl, int nt, const float *img, float2 *S, const float2 *twx,
                        cudaStream_t s, bool first)
{
    const SxOps *o = sx_ops(g.P[0]);
    if (!o) return cudaErrorInvalidValue;
    const int rows = tile_max(tl, nt, [](const SepTile &t) { return t.a[1].nq * t.a[2].nq; });
    return o->ratio(g, tl, nt, sep_row_ctas(g.P[0], rows), img, S, aligned8(img), twx, s, first);
}

cudaError_t sep_x_update(const SepGeom &g, const SepTiles &tl, int nt, int epi, const SepUpd &u, const float2 *S,
                         const float2 *twx, cudaStream_t s, bool first)
{
    const SxOps *o = sx_ops(g.P[0]);
    if (!o) return cudaErrorInvalidValue;
    const int rows = tile_max(tl, nt, [](const SepTile &t) { return t.a[1].nw * t.a[2].nw; });
    const bool vec = aligned8(u.psi) && aligned8(u.dst) && aligned8(u.weight[0]);
    return o->update(g, tl, nt, sep_row_ctas(g.P[0], rows), epi, u, S, vec, twx, s, first);
}

cudaError_t sep_y_fwd(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, const int kd[3], float2 *S,
                      const float2 *twy, cudaStream_t s)
{
    const YzOps *o = yz_ops(g.P[1]);
    if (!o) return cudaErrorInvalidValue;
    const int planes = map == SEP_MIRROR ? tile_max(tl, nt, [](const SepTile &t) { return t.a[2].nv; })
                       : map == SEP_FILL ? tile_max(tl, nt, [](const SepTile &t) { return t.a[2].nq; })
                                         : kd[2];
    return o->y_fwd(g, sl, tl, nt, map, kd ? kd[1] : 0, kd ? kd[2] : 0, S, twy, s, planes);
}

cudaError_t sep_y_inv(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int out_w, float2 *S, const float2 *twy,
                      cudaStream_t s)
{
    const YzOps *o = yz_ops(g.P[1]);
    if (!o) return cudaErrorInvalidValue;
    const int planes = tile_max(tl, nt, [out_w](const SepTile &t) { return out_w ? t.a[2].nw : t.a[2].nq; });
    return o->y_inv(g, sl, tl, nt, out_w, S, twy, s, planes);
}

cudaError_t sep_z(const SepGeom &g, const SepSlab &sl, const SepTiles &tl, int nt, int map, int out_w, const int kd[3], const float2 *src,
                  float2 *dst, const float2 *K, const float2 *twz, cudaStream_t s)
{
    const YzOps *o = yz_ops(g.P[2]);
    if (!o) return cudaErrorInvalidValue;
    return o->z(g, sl, tl, nt, map, out_w, kd ? kd[2] : 0, src, dst, K, twz, s);
}

}  // namespace mvr
