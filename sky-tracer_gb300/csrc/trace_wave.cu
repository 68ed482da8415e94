// trace_wave.cu — the launch sequence of the wavefront tracer: prepare (zero
// the sums of jobs that do not accumulate, reset the work counter), trace
// (trace_wave.cuh, or trace_ray.cuh for small renders, instantiated per
// tracking mode in trace_wave_*.cu and trace_ray_*.cu) and finalize (film, XYZ,
// variance, linear sRGB of every job).

#include <algorithm>

#include "trace_kernels.h"

namespace sky {
namespace {

// Zero the sums of every job that does not accumulate (blockIdx.y = job) and
// reset the work counter.
__global__ void __launch_bounds__(256) wave_prepare_kernel(const DevJob* __restrict__ jobs,
                                                           unsigned long long* __restrict__ work_counter) {
    const DevJob& J = jobs[blockIdx.y];
    if (blockIdx.x == 0u && blockIdx.y == 0u && threadIdx.x == 0u) *work_counter = 0ull;
    if (J.accumulate) return;
    double* sum = J.cell_sum;
    double* sq = J.cell_sumsq;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < J.cell_count;
         i += uint64_t(gridDim.x) * blockDim.x) {
        sum[i] = 0.0;
        if (sq) sq[i] = 0.0;
    }
}

}  // namespace

// A launch goes to the ray loop (trace_ray.cuh) rather than to the stage
// queues (trace_wave.cuh) where it has so few chains per lane of the chip
// (1024 lanes per SM) that its longest chains decide its time.  Measured with
// both kernels (ms, ray loop against queues):
//   merged layers      one species: 3.1 M chains 0.63 / 0.65, 4.2 M 0.79 / 0.75: 24 per lane;
//                      four: 4.0 M 1.47 / 1.60, 5.4 M 1.86 / 1.81: 34 per lane
//   residual carry     one species: 131 k 0.52 / 0.68, 262 k 0.63 / 0.62, 524 k 0.82 / 0.70: 2 per lane;
//                      four (64x32, 41 bands): 0.32 M 0.95 / 1.08, 0.47 M 1.12 / 1.15, 0.62 M 1.28 / 1.29,
//                      0.78 M 1.45 / 1.35: 5 per lane
//   segment restart    0.67 M 1.25 / 1.34, 1.0 M 1.63 / 1.12: 5 per lane
uint64_t wave_queue_chains(uint32_t tracking, uint32_t aerosol_species, int sms) {
    const uint64_t per_lane = tracking == SKY_TRACKING_SEGMENT_RESTART  ? 5u
                              : tracking == SKY_TRACKING_RESIDUAL_CARRY ? (aerosol_species == 1u ? 2u : 5u)
                              : aerosol_species == 1u                   ? 24u
                                                                        : 34u;
    return per_lane * 1024u * uint64_t(sms);
}

cudaError_t launch_trace_wave(const WaveLaunch& asked, cudaStream_t stream) {
    WaveLaunch w = asked;
    if (w.num_jobs == 0u || w.num_jobs > 65535u || w.total_cells == 0u) return cudaErrorInvalidValue;
    const uint32_t xblocks =
        uint32_t(std::min<uint64_t>((uint64_t(w.max_job_cells) + 255u) / 256u, 1024u));
    wave_prepare_kernel<<<dim3(std::max(xblocks, 1u), w.num_jobs), 256, 0, stream>>>(w.jobs, w.work_counter);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&w.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    const bool small = w.total_chains < wave_queue_chains(w.tracking, w.aerosol_species, w.sms);
    switch (w.tracking) {
        case SKY_TRACKING_SEGMENT_RESTART:
            e = small ? launch_ray_segment_restart(w, stream) : launch_wave_segment_restart(w, stream);
            break;
        case SKY_TRACKING_RESIDUAL_CARRY:
            e = small ? launch_ray_residual_carry(w, stream) : launch_wave_residual_carry(w, stream);
            break;
        case SKY_TRACKING_MERGED_LAYERS:
            e = small ? launch_ray_merged_layers(w, stream) : launch_wave_merged_layers(w, stream);
            break;
        default: return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    return launch_finalize_jobs(w.scene, w.jobs, w.num_jobs, w.total_cells, stream);
}

}  // namespace sky
