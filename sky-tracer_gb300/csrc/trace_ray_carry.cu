// trace_ray_carry.cu — the small-render kernels of residual-carry tracking.

#include "trace_ray.cuh"

namespace sky {

cudaError_t launch_ray_residual_carry(const WaveLaunch& w, cudaStream_t stream) {
    return ray::launch_ray_tracking<SKY_TRACKING_RESIDUAL_CARRY>(w, stream);
}

}  // namespace sky
