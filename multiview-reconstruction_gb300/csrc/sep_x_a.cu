// x passes of the separable transforms (sep_x.cuh): lengths 64, 96, 128, 160, 192.
#include "sep_x.cuh"

namespace mvr {

const SxOps *sx_ops_a(int n)
{
    switch (n) {
    case 64: return Sx<2>::ops();
    case 96: return Sx<3>::ops();
    case 128: return Sx<4>::ops();
    case 160: return Sx<5>::ops();
    case 192: return Sx<6>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
