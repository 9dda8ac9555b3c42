// y and z passes of the separable transforms (sep_yz.cuh): lengths 256, 288, 320, 360.
#include "sep_yz.cuh"

namespace mvr {

const YzOps *yz_ops_c(int n)
{
    switch (n) {
    case 256: return Yz<16, 16>::ops();
    case 288: return Yz<16, 18>::ops();
    case 320: return Yz<16, 20>::ops();
    case 360: return Yz<18, 20>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
