// fi_resident_large.cu -- the resident step kernel with the radix sequences of the square
// grids 256, 350, 512 and 1024 compiled in.
#include "fi_resident.cuh"

namespace fi {

const void* resident_large(int seq, int all) {
    if (all) {
        switch (seq) {
            case 2288: return (const void*)k_resident<2288, 2288, 1>;
            case 5527: return (const void*)k_resident<5527, 5527, 1>;
            default: return nullptr;
        }
    }
    switch (seq) {
        case 888: return (const void*)k_resident<888, 888, 0>;
        case 8484: return (const void*)k_resident<8484, 8484, 0>;
        default: return nullptr;
    }
}

}  // namespace fi
