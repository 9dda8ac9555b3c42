// y and z passes of the separable transforms (sep_yz.cuh): lengths 32, 48, 64, 80, 96, 112.
#include "sep_yz.cuh"

namespace mvr {

const YzOps *yz_ops_a(int n)
{
    switch (n) {
    case 32: return Yz<4, 8>::ops();
    case 48: return Yz<6, 8>::ops();
    case 64: return Yz<8, 8>::ops();
    case 80: return Yz<8, 10>::ops();
    case 96: return Yz<8, 12>::ops();
    case 112: return Yz<8, 14>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
