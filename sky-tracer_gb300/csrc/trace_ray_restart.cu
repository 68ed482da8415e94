// trace_ray_restart.cu — the small-render kernels of segment-restart tracking.

#include "trace_ray.cuh"

namespace sky {

cudaError_t launch_ray_segment_restart(const WaveLaunch& w, cudaStream_t stream) {
    return ray::launch_ray_tracking<SKY_TRACKING_SEGMENT_RESTART>(w, stream);
}

}  // namespace sky
