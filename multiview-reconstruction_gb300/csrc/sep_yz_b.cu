// y and z passes of the separable transforms (sep_yz.cuh): lengths 128, 144, 160, 192, 224.
#include "sep_yz.cuh"

namespace mvr {

const YzOps *yz_ops_b(int n)
{
    switch (n) {
    case 128: return Yz<8, 16>::ops();
    case 144: return Yz<12, 12>::ops();
    case 160: return Yz<10, 16>::ops();
    case 192: return Yz<12, 16>::ops();
    case 224: return Yz<14, 16>::ops();
    default: return nullptr;
    }
}

}  // namespace mvr
