// trace_ray_merged.cu — the small-render kernels of merged-layer tracking.

#include "trace_ray.cuh"

namespace sky {

cudaError_t launch_ray_merged_layers(const WaveLaunch& w, cudaStream_t stream) {
    return ray::launch_ray_tracking<SKY_TRACKING_MERGED_LAYERS>(w, stream);
}

}  // namespace sky
