// x passes of the separable transforms (sep_x.cuh): lengths 224, 256, 288, 320.
#include "sep_x.cuh"

namespace mvr {

const SxOps *sx_ops_b(int n)
{
    switch (n) {
    case 224: return Sx<7>::ops();
    case 256: return Sx<8>::ops();
    case 288: return Sx<9>::ops();
    case 320: return Sx<10>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
