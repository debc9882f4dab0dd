// fi_resident_small.cu -- the resident step kernel with the radix sequences of the square
// grids 64, 96, 128 and 192 compiled in.
#include "fi_resident.cuh"

namespace fi {

const void* resident_small(int seq) {
    switch (seq) {
        case 444: return (const void*)k_resident<444, 444, 1>;
        case 834: return (const void*)k_resident<834, 834, 1>;
        case 484: return (const void*)k_resident<484, 484, 1>;
        case 838: return (const void*)k_resident<838, 838, 1>;
        default: return nullptr;
    }
}

}  // namespace fi
