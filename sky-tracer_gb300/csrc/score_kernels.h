// score_kernels.h — launcher of the combination-score kernels (score.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace sky {

constexpr uint32_t kScoreHistBins = 2048;  // widest radix-selection pass: 11 bits
constexpr uint32_t kScoreGroup = 4;        // combinations of a block of the distances
constexpr uint32_t kScoreTargets = 5;      // p50, p90, p95, p99, max

// One combination's sums over its finite distances, and the selection of its
// order statistics: after the last pass prefix[t] holds the bits of target t.
struct ScoreState {
    double sum, sum_sq;
    uint64_t count;
    uint64_t rank[kScoreTargets];
    uint32_t prefix[kScoreTargets];
    uint32_t _pad;
};

struct ScoreLaunch {
    const float* bands;           // [..][samples]
    uint64_t samples;
    const float* ref_lab;         // [samples][3]
    float inv_scale;
    const uint32_t* combo_bands;  // [combos][channels]
    const float* combo_xyz;       // [combos][channels][3]
    uint32_t combos, channels;
    float* dist;                  // [combos][samples]: Oklab distances, NaN when not finite
    ScoreState* state;            // [combos], zeroed by the caller
    uint32_t* hist;               // [combos][kScoreTargets][kScoreHistBins], zeroed by the caller (left zeroed)
    uint32_t sms;
};
cudaError_t launch_score(const ScoreLaunch& w, cudaStream_t stream);

// The reference's scale (the 99th percentile of its finite Y, at least 1e-12)
// and the state of its selection.
struct ScaleState {
    double scale;
    uint64_t count, rank, prefix;
    uint32_t ended;  // blocks of a pass that are done
    uint32_t _pad;
};
// state and hist [kScoreHistBins] zeroed by the caller (hist left zeroed).
cudaError_t launch_reference_scale(const double* ref_xyz, uint64_t samples, ScaleState* state, uint32_t* hist,
                                   uint32_t sms, cudaStream_t stream);
// ref_lab [samples][3]: Oklab of ref_xyz / state->scale.
cudaError_t launch_reference_lab(const double* ref_xyz, uint64_t samples, const ScaleState* state, float* ref_lab,
                                 cudaStream_t stream);

}  // namespace sky
