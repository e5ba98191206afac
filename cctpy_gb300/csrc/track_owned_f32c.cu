// The owned schedule's FP32c kernels (track_owned.cuh).
#include "track_owned.cuh"

namespace cctgpu {

TrackKernel owned_kernel_f32c(int G, bool few) {
    switch (G) {
        case 16: return few ? track_owned_kernel<false, 16> : track_owned_kernel<false, 16, false, true>;
        case 32: return few ? track_owned_kernel<false, 32> : track_owned_kernel<false, 32, false, true>;
        case 64: return few ? track_owned_kernel<false, 64> : track_owned_kernel<false, 64, false, true>;
        case 128: return few ? track_owned_kernel<false, 128> : track_owned_kernel<false, 128, false, true>;
        default: return few ? track_owned_kernel<false, 256> : track_owned_kernel<false, 256, false, true>;
    }
}

}  // namespace cctgpu
