// y and z passes of the separable transforms (sep_yz.cuh): lengths 400, 432, 480, 576.
#include "sep_yz.cuh"

namespace mvr {

const YzOps *yz_ops_d(int n)
{
    switch (n) {
    case 400: return Yz<20, 20>::ops();
    case 432: return Yz<18, 24>::ops();
    case 480: return Yz<20, 24>::ops();
    case 576: return Yz<24, 24>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
