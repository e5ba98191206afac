// The owned schedule's FP64 kernels (track_owned.cuh).
#include "track_owned.cuh"

namespace cctgpu {

TrackKernel owned_kernel_f64(int G) {
    return G == 8 ? track_owned_kernel<true, 8> : G == 16 ? track_owned_kernel<true, 16> : track_owned_kernel<true, 32>;
}

}  // namespace cctgpu
