// The owned schedule's FP32c kernels (track_owned.cuh).
#include "track_owned.cuh"

namespace cctgpu {

TrackKernel owned_kernel_f32c(int G) {
    switch (G) {
        case 16: return track_owned_kernel<false, 16>;
        case 32: return track_owned_kernel<false, 32>;
        case 64: return track_owned_kernel<false, 64>;
        case 128: return track_owned_kernel<false, 128>;
        default: return track_owned_kernel<false, 256>;
    }
}

}  // namespace cctgpu
