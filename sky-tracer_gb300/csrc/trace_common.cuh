// trace_common.cuh — what the two persistent tracing kernels (trace_wave.cuh,
// trace_ray.cuh) share: the lookup of a lane's job and the medium tables
// staged in a block's shared memory.

#pragma once

#include "sky_device.cuh"
#include "trace_kernels.h"

namespace sky {
namespace wave {

constexpr uint32_t kFull = 0xffffffffu;
// Default backstop on the loop iterations of one warp (SkyTuning.iteration_limit
// overrides it).  Beyond it the warp sets status bit 2 and returns.
constexpr uint32_t kMaxIterations = 1u << 31;

// The launch constants and the sun frame of a lane's job: kernel parameters
// when the launch holds one job, the job table otherwise.
template <bool kSingle>
__device__ __forceinline__ const DevLaunch& job_launch(const DevLaunch& L0, const DevJob* jobs, uint32_t job) {
    if constexpr (kSingle) return L0;
    else return jobs[job].L;
}
template <bool kSingle>
__device__ __forceinline__ const DevScene& job_scene(const DevScene& S0, const DevJob* jobs, uint32_t job) {
    if constexpr (kSingle) return S0;
    else return jobs[job].S;
}

// Bytes of shared memory that stage_medium() fills: the band-independent knot
// profile (48 B per knot), the per-band constants (32 B per band) and aerosol
// optics (32 B per band), the union knots and the knot finder.
__host__ __device__ inline size_t staged_medium_bytes(uint32_t knots, uint32_t bands) {
    return size_t(knots) * sizeof(DevProfileKnot) + size_t(bands) * sizeof(DevBand) +
           size_t(bands) * kSpecies * sizeof(SkyAerosolOptics) + size_t(knots) * sizeof(float) +
           size_t(kFinderCells) * sizeof(uint16_t);
}

// Copy the medium tables every collision and NEE evaluation reads into the
// block's shared memory (once per block, before the loop), and return the
// view of them.  The per-band extinction rows and the phase tables stay in
// global memory, read through the L1 cache.
__device__ __forceinline__ Medium stage_medium(const DevScene& S, unsigned char* smem) {
    DevProfileKnot* profile = reinterpret_cast<DevProfileKnot*>(smem);
    DevBand* bands = reinterpret_cast<DevBand*>(profile + S.knot_count);
    SkyAerosolOptics* optics = reinterpret_cast<SkyAerosolOptics*>(bands + S.band_count);
    float* knot_z = reinterpret_cast<float*>(optics + S.band_count * kSpecies);
    uint16_t* finder = reinterpret_cast<uint16_t*>(knot_z + S.knot_count);
    // 4-byte words throughout (every table is a multiple of 4 bytes; the finder's 512 halves are 256 words)
    auto copy = [](void* dst, const void* src, size_t bytes) {
        uint32_t* d = static_cast<uint32_t*>(dst);
        const uint32_t* s = static_cast<const uint32_t*>(src);
        for (size_t i = threadIdx.x; i < bytes / 4u; i += blockDim.x) d[i] = __ldg(s + i);
    };
    copy(profile, S.profile, size_t(S.knot_count) * sizeof(DevProfileKnot));
    copy(bands, S.bands, size_t(S.band_count) * sizeof(DevBand));
    copy(optics, S.optics, size_t(S.band_count) * kSpecies * sizeof(SkyAerosolOptics));
    copy(knot_z, S.knot_z, size_t(S.knot_count) * sizeof(float));
    copy(finder, S.finder, size_t(kFinderCells) * sizeof(uint16_t));
    __syncthreads();
    return Medium{knot_z, finder, profile, bands, optics};
}

}  // namespace wave
}  // namespace sky
