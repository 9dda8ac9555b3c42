// x passes of the separable transforms (sep_x.cuh): lengths 384, 448, 512, 576.
#include "sep_x.cuh"

namespace mvr {

const SxOps *sx_ops_c(int n)
{
    switch (n) {
    case 384: return Sx<12>::ops();
    case 448: return Sx<14>::ops();
    case 512: return Sx<16>::ops();
    case 576: return Sx<18>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
