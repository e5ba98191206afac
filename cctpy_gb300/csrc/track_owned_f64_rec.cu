// The owned schedule's FP64 kernels for the adjoint's forward (track_owned.cuh).
#include "track_owned.cuh"

namespace cctgpu {

TrackKernel owned_kernel_f64_rec(int G) {
    return G == 8 ? track_owned_kernel<true, 8, true> : G == 16 ? track_owned_kernel<true, 16, true> : track_owned_kernel<true, 32, true>;
}

}  // namespace cctgpu
