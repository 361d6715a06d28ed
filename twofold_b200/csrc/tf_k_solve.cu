// Step preparation and the substep (tf_kernels.cuh), compiled on their own.
#include "tf_kernels.cuh"
#include "tf_launch.h"

namespace tfb {

const void* solveKernels(int id) {
    switch (id) {
        case kKPrepare: return (const void*)k_prepare<false>;
        case kKPrepareBig: return (const void*)k_prepare<true>;
        case kKSubstep: return (const void*)k_substep<false, false>;
        case kKSubstepJoints: return (const void*)k_substep<true, false>;
        case kKSubstepRooms: return (const void*)k_substep<false, true>;
        case kKSubstepRoomsJoints: return (const void*)k_substep<true, true>;
        default: return nullptr;
    }
}

}  // namespace tfb
