// score.cu — the wavelength optimizer's combination score on the GPU.
//
// sky-wavelength-optimizer scores a combination of primary bands by
// rebuilding every sample's XYZ from the selected bands
// (xyz = sum_ch band[idx_ch][s] * c_ch, c_ch = weight_nm / band_width * CIE),
// mapping it and the full-spectrum reference to Oklab at a common scale, and
// summarising the per-sample distances: mean, RMS, the p50/p90/p95/p99
// percentiles of the sorted finite distances (element round((n-1) q)) and
// the maximum; score = rmse + 0.25 p95 (main.rs:414-488, 1121-1156).
//
// Here one launch computes every sample's distance for a batch of
// combinations, and the percentiles are exact order statistics found by radix
// selection over the distances' IEEE bits (non-negative floats order like
// their bit patterns): an 11-bit, an 11-bit and a 10-bit histogram pass, with
// the picks between them made on the device.
//
// What bounds it: FP32 and special-function issue of the distances (three cube
// roots each).  Two things stood above that bound and are gone.  FP64 runs at
// 2 operations per clock and SM, and reducing every 256 distances to FP64
// block sums took 15 of them per distance: a thread now sums its distances and
// their squares exactly in pairs of floats and adds 32 of them at a time to
// FP64.  And each of a combination's five order statistics read all distances
// three times: the first histogram is now taken while the distances are made,
// the others from one reading for all five, of a buffer that stays in L2.
// 655 360 samples x 128 combinations of 4 bands: 5.9 ms of kernels and four
// round trips to the host -> 1.3 ms (distances 0.80, histograms 0.36, picks 0.13)
// and one.  The reference's scale and Oklab (0.18 ms here) took 33 ms on the host.
// One distance at a time per thread, one target's scan after the other in the
// picks, and one warp for the scale's: 1.8 and 0.34 ms.

#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstdint>

#include "score_kernels.h"

namespace sky {
namespace {

__device__ __forceinline__ float signed_cbrt(float x) {
    const float a = fabsf(x);
    const float r = a > 0.0f ? exp2f(__log2f(a) * (1.0f / 3.0f)) : a;  // keeps 0 and NaN
    return copysignf(r, x);
}

// Oklab of XYZ (Ottosson's published matrices), main.rs:1121-1130.
__device__ __forceinline__ void xyz_to_oklab(float x, float y, float z, float lab[3]) {
    const float l = signed_cbrt(0.8189330101f * x + 0.3618667424f * y - 0.1288597137f * z);
    const float m = signed_cbrt(0.0329845436f * x + 0.9293118715f * y + 0.0361456387f * z);
    const float s = signed_cbrt(0.0482003018f * x + 0.2643662691f * y + 0.6338517070f * z);
    lab[0] = 0.2104542553f * l + 0.7936177850f * m - 0.0040720468f * s;
    lab[1] = 1.9779984951f * l - 2.4285922050f * m + 0.4505937099f * s;
    lab[2] = 0.0259040371f * l + 0.7827717662f * m - 0.8086757660f * s;
}

// Combinations of a block, and samples of a thread in a tile.
constexpr uint32_t kCombos = kScoreGroup, kSamples = 4;
constexpr uint32_t kTile = 256u * kSamples;

// A sum kept as an unevaluated pair of floats.  Each addition's rounding error
// is exact (Knuth's two-sum) and goes to `lo`: 32 terms are off by less than
// 32 x 2^-47, then they join an FP64 sum.
struct PairSum {
    float hi, lo;
    __device__ __forceinline__ void add(float v, float rest) {
        const float t = __fadd_rn(hi, v), b = __fsub_rn(t, hi);
        lo = __fadd_rn(lo, __fadd_rn(__fadd_rn(__fsub_rn(hi, __fsub_rn(t, b)), __fsub_rn(v, b)), rest));
        hi = t;
    }
    __device__ __forceinline__ double take() {
        const double d = double(hi) + double(lo);
        hi = lo = 0.0f;
        return d;
    }
};

// Bits of the distances from 2^-40 on and below 2^60, whose squares a PairSum holds: a
// square's rounding error, a multiple of its exponent's 2^-46, is no denormal (those are
// flushed to 0), and 32 squares' sum is finite.  The others' go to FP64.
constexpr uint32_t kLeastSquare = (127u - 40u) << 23, kMostSquare = (127u + 60u) << 23;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Distances of kCombos combinations from blockIdx.y on, tiles of samples from
// blockIdx.x on; FP64 sum and sum of squares and count of the finite ones, and
// the histogram of their top 11 bits.
__global__ void __launch_bounds__(256) distance_kernel(const float* __restrict__ bands, uint64_t samples,
                                                       const float* __restrict__ ref_lab, float inv_scale,
                                                       const uint32_t* __restrict__ combo_bands,
                                                       const float* __restrict__ combo_xyz, uint32_t combos,
                                                       uint32_t channels, float* __restrict__ dist,
                                                       ScoreState* __restrict__ state, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kCombos][kScoreHistBins];
    for (uint32_t i = threadIdx.x; i < kCombos * kScoreHistBins; i += blockDim.x) (&h[0][0])[i] = 0u;
    __syncthreads();
    const uint32_t c0 = blockIdx.y * kCombos;
    PairSum s1[kCombos], s2[kCombos];
    double t1[kCombos], t2[kCombos];
    uint32_t n[kCombos];
#pragma unroll
    for (uint32_t k = 0; k < kCombos; ++k) {
        s1[k] = s2[k] = PairSum{0.0f, 0.0f};
        t1[k] = t2[k] = 0.0;
        n[k] = 0u;
    }
    uint32_t pending = 0u;
    for (uint64_t tile = uint64_t(blockIdx.x) * kTile; tile < samples; tile += uint64_t(gridDim.x) * kTile) {
        uint64_t at[kSamples];
        float l0[kSamples], a0[kSamples], b0[kSamples];
#pragma unroll
        for (uint32_t j = 0; j < kSamples; ++j) {
            at[j] = tile + j * 256u + threadIdx.x;
            const bool in = at[j] < samples;
            l0[j] = in ? __ldg(ref_lab + at[j] * 3) : 0.0f;
            a0[j] = in ? __ldg(ref_lab + at[j] * 3 + 1) : 0.0f;
            b0[j] = in ? __ldg(ref_lab + at[j] * 3 + 2) : 0.0f;
        }
#pragma unroll
        for (uint32_t k = 0; k < kCombos; ++k) {
            const uint32_t c = c0 + k;
            if (c >= combos) break;  // uniform over the block
            float x[kSamples] = {}, y[kSamples] = {}, z[kSamples] = {};
            for (uint32_t ch = 0; ch < channels; ++ch) {
                const float* band = bands + uint64_t(__ldg(combo_bands + size_t(c) * channels + ch)) * samples;
                const float* w = combo_xyz + (size_t(c) * channels + ch) * 3u;
                const float wx = __ldg(w), wy = __ldg(w + 1), wz = __ldg(w + 2);
#pragma unroll
                for (uint32_t j = 0; j < kSamples; ++j) {
                    const float v = at[j] < samples ? __ldg(band + at[j]) : 0.0f;
                    x[j] = fmaf(v, wx, x[j]);
                    y[j] = fmaf(v, wy, y[j]);
                    z[j] = fmaf(v, wz, z[j]);
                }
            }
#pragma unroll
            for (uint32_t j = 0; j < kSamples; ++j) {
                if (at[j] >= samples) continue;
                float lab[3];
                xyz_to_oklab(x[j] * inv_scale, y[j] * inv_scale, z[j] * inv_scale, lab);
                const float dl = lab[0] - l0[j], da = lab[1] - a0[j], db = lab[2] - b0[j];
                float e = sqrtf(dl * dl + da * da + db * db);
                const uint32_t bits = __float_as_uint(e);
                if (bits - kLeastSquare < kMostSquare - kLeastSquare) {
                    const float q = __fmul_rn(e, e);
                    s1[k].add(e, 0.0f);
                    s2[k].add(q, __fmaf_rn(e, e, -q));
                    ++n[k];
                    atomicAdd(&h[k][bits >> 21], 1u);
                } else if (isfinite(e)) {
                    if (e != 0.0f) {
                        t1[k] += double(e);
                        t2[k] += double(e) * double(e);
                    }
                    ++n[k];
                    atomicAdd(&h[k][bits >> 21], 1u);
                } else {
                    e = __int_as_float(0x7fffffff);  // NaN: not counted, not selected
                }
                dist[size_t(c) * samples + at[j]] = e;
            }
        }
        if (++pending == 32u / kSamples) {
            pending = 0u;
#pragma unroll
            for (uint32_t k = 0; k < kCombos; ++k) {
                t1[k] += s1[k].take();
                t2[k] += s2[k].take();
            }
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kCombos; ++k) {
        const double sum = warp_sum(t1[k] + s1[k].take()), sq = warp_sum(t2[k] + s2[k].take());
        const uint32_t count = __reduce_add_sync(0xffffffffu, n[k]);
        if ((threadIdx.x & 31u) == 0u && c0 + k < combos && count) {
            ScoreState& S = state[c0 + k];
            atomicAdd(&S.sum, sum);
            atomicAdd(&S.sum_sq, sq);
            atomicAdd(reinterpret_cast<unsigned long long*>(&S.count), (unsigned long long)count);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kCombos * kScoreHistBins; i += blockDim.x) {
        const uint32_t k = i / kScoreHistBins, bin = i % kScoreHistBins;
        if (h[k][bin]) atomicAdd(hist + size_t(c0 + k) * kScoreTargets * kScoreHistBins + bin, h[k][bin]);
    }
}

// Histograms of the next `width` bits of combination blockIdx.y's distances,
// one for each of its targets' prefixes (the bits above `shift + width`).
// Targets with the same prefix share the first one's.  A thread reads four
// distances at a time (one at a time, the last digit's reading, which finds almost
// none of its prefixes, took 67 us for 65 MB of L2).
__global__ void __launch_bounds__(256) select_hist_kernel(const float* __restrict__ dist, uint64_t samples,
                                                          const ScoreState* __restrict__ state, uint32_t shift,
                                                          uint32_t width, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kScoreTargets][kScoreHistBins];
    const uint32_t c = blockIdx.y, bins = 1u << width, top = shift + width;
    const ScoreState& S = state[c];
    if (S.count == 0u) return;
    uint32_t prefix[kScoreTargets];
#pragma unroll
    for (uint32_t t = kScoreTargets; t-- > 0u;)  // 0xffffffff: no distance has it
        prefix[t] = t && S.prefix[t] == S.prefix[t - 1u] ? 0xffffffffu : S.prefix[t];
    for (uint32_t i = threadIdx.x; i < kScoreTargets * kScoreHistBins; i += blockDim.x) (&h[0][0])[i] = 0u;
    __syncthreads();
    const float* row = dist + size_t(c) * samples;
    for (uint64_t tile = uint64_t(blockIdx.x) * kTile; tile < samples; tile += uint64_t(gridDim.x) * kTile) {
        uint32_t bits[kSamples];
#pragma unroll
        for (uint32_t j = 0; j < kSamples; ++j) {
            const uint64_t s = tile + j * 256u + threadIdx.x;
            bits[j] = s < samples ? __float_as_uint(__ldg(row + s)) : 0x7fffffffu;  // NaN: above every prefix
        }
#pragma unroll
        for (uint32_t j = 0; j < kSamples; ++j) {
            const uint32_t above = bits[j] >> top, digit = (bits[j] >> shift) & (bins - 1u);
#pragma unroll
            for (uint32_t t = 0; t < kScoreTargets; ++t)
                if (above == prefix[t]) atomicAdd(&h[t][digit], 1u);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kScoreTargets * bins; i += blockDim.x) {
        const uint32_t t = i >> width, bin = i & (bins - 1u);
        if (h[t][bin]) atomicAdd(hist + (size_t(c) * kScoreTargets + t) * kScoreHistBins + bin, h[t][bin]);
    }
}

// Of each target of combination blockIdx.x, the digit that holds its rank: a
// block scan of its histogram (which is cleared for the next pass), the rank
// within the digit, and the prefix with the digit appended.
__global__ void __launch_bounds__(256) select_pick_kernel(ScoreState* __restrict__ state, uint32_t first,
                                                          uint32_t width, uint32_t* __restrict__ hist) {
    constexpr uint32_t kPer = kScoreHistBins / 256u;
    __shared__ uint64_t warp_total[kScoreTargets][8];
    ScoreState& S = state[blockIdx.x];
    const uint64_t count = S.count;
    if (count == 0u) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // percentile_sorted: element round((n - 1) q), half away from 0
    const double quantile[kScoreTargets] = {0.50, 0.90, 0.95, 0.99, 1.0};
    uint32_t prefix[kScoreTargets];
    uint64_t rank[kScoreTargets];
#pragma unroll
    for (uint32_t t = 0; t < kScoreTargets; ++t) {
        prefix[t] = S.prefix[t];
        rank[t] = first ? uint64_t(floor(double(count - 1u) * quantile[t] + 0.5)) : S.rank[t];
    }
    // all rows' loads under way at once, 16 bytes each
    uint32_t own[kScoreTargets][kPer];
    uint64_t upto[kScoreTargets];
    uint32_t owner = 0u;  // the prefixes ascend with the targets' ranks: equal ones are neighbours
    static_assert(kPer == 8u, "two 16-byte words of bins per thread");
    uint4* const rows = reinterpret_cast<uint4*>(hist + size_t(blockIdx.x) * kScoreTargets * kScoreHistBins) + tid * 2u;
#pragma unroll
    for (uint32_t t = 0; t < kScoreTargets; ++t) {
        if (t && !first && prefix[t] != prefix[t - 1u]) owner = t;
#pragma unroll
        for (uint32_t q = 0; q < 2u; ++q) {
            const uint4 v = rows[owner * (kScoreHistBins / 4u) + q];
            own[t][q * 4u] = v.x;
            own[t][q * 4u + 1u] = v.y;
            own[t][q * 4u + 2u] = v.z;
            own[t][q * 4u + 3u] = v.w;
        }
    }
#pragma unroll
    for (uint32_t t = 0; t < kScoreTargets; ++t) {
        upto[t] = 0u;
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) upto[t] += own[t][i];
        // this thread's bins, which it has read
        rows[t * (kScoreHistBins / 4u)] = rows[t * (kScoreHistBins / 4u) + 1u] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (uint32_t t = 0; t < kScoreTargets; ++t) {
        const uint64_t mine = upto[t];
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint64_t v = __shfl_up_sync(0xffffffffu, upto[t], o);
            if (lane >= o) upto[t] += v;
        }
        if (lane == 31u) warp_total[t][warp] = upto[t];
        upto[t] -= mine;
    }
    __syncthreads();  // and the state is read by all before one of them writes it
#pragma unroll
    for (uint32_t t = 0; t < kScoreTargets; ++t) {
        uint64_t below = upto[t];
        for (uint32_t w = 0; w < warp; ++w) below += warp_total[t][w];
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            if (rank[t] >= below && rank[t] - below < own[t][i]) {  // one thread has it
                S.rank[t] = rank[t] - below;
                S.prefix[t] = (prefix[t] << width) | (tid * kPer + i);
            }
            below += own[t][i];
        }
    }
}

// ---- the reference: its scale and its Oklab ------------------------------------

// Doubles in the order of their values, as unsigned keys.
__device__ __forceinline__ uint64_t order_key(double v) {
    const uint64_t b = uint64_t(__double_as_longlong(v));
    return b >> 63 ? ~b : b | (uint64_t(1) << 63);
}
__device__ __forceinline__ double key_value(uint64_t k) {
    return __longlong_as_double((long long)(k >> 63 ? k & ~(uint64_t(1) << 63) : ~k));
}

// One digit of the radix selection of element round((n - 1) 0.99) of the finite
// Y (main.rs:343, :1150-1156): the histogram of the keys that share the digits
// above, and, by the block that ends last, the digit's pick.  The first pass
// also counts the finite ones.
__global__ void __launch_bounds__(256) scale_select_kernel(const double* __restrict__ ref_xyz, uint64_t samples,
                                                           uint32_t shift, uint32_t width, uint32_t first,
                                                           ScaleState* __restrict__ state,
                                                           uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kScoreHistBins];
    __shared__ uint32_t last;
    __shared__ uint64_t warp_total[8];
    const uint32_t bins = 1u << width, top = shift + width;
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) h[i] = 0u;
    const uint64_t prefix = first ? 0u : state->prefix;
    __syncthreads();
    uint32_t n = 0u;
    for (uint64_t tile = uint64_t(blockIdx.x) * kTile; tile < samples; tile += uint64_t(gridDim.x) * kTile) {
        double y[kSamples];
#pragma unroll
        for (uint32_t j = 0; j < kSamples; ++j) {
            const uint64_t s = tile + j * 256u + threadIdx.x;
            y[j] = s < samples ? ref_xyz[s * 3 + 1] : CUDART_INF;
        }
#pragma unroll
        for (uint32_t j = 0; j < kSamples; ++j) {
            if (!isfinite(y[j])) continue;
            const uint64_t key = order_key(y[j]);
            if (!first && (key >> top) != prefix) continue;
            ++n;
            atomicAdd(&h[uint32_t(key >> shift) & (bins - 1u)], 1u);
        }
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (first && (threadIdx.x & 31u) == 0u && n)
        atomicAdd(reinterpret_cast<unsigned long long*>(&state->count), (unsigned long long)n);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x)
        if (h[i]) atomicAdd(hist + i, h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0u) last = atomicAdd(&state->ended, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // a block scan of the digit's histogram, bins / 256 neighbouring bins to a thread
    // (32 bins at a time by one warp: 28 of a pass's 45 us)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, per = bins / 256u;
    const uint64_t count = *reinterpret_cast<volatile uint64_t*>(&state->count);
    const uint64_t rank = first ? (count ? uint64_t(floor(double(count - 1u) * 0.99 + 0.5)) : 0u) : state->rank;
    for (uint32_t i = tid; i < bins; i += 256u) {
        h[i] = *reinterpret_cast<volatile uint32_t*>(hist + i);
        hist[i] = 0u;
    }
    __syncthreads();
    uint64_t mine = 0u;
    for (uint32_t i = 0; i < per; ++i) mine += h[tid * per + i];
    uint64_t upto = mine;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint64_t v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    if (lane == 31u) warp_total[warp] = upto;
    __syncthreads();  // the rank is read by all before one of them writes it
    uint64_t below = upto - mine;
    for (uint32_t w = 0; w < warp; ++w) below += warp_total[w];
    for (uint32_t i = 0; i < per; ++i) {
        const uint32_t own = h[tid * per + i];
        if (rank >= below && rank - below < own) {  // one thread has it
            state->prefix = (prefix << width) | (tid * per + i);
            state->rank = rank - below;
        }
        below += own;
    }
    if (tid == 0u) state->ended = 0u;
}

// The scale: the selected Y, at least 1e-12 (also without a finite one).
__global__ void scale_value_kernel(ScaleState* __restrict__ state) {
    state->scale = state->count ? fmax(key_value(state->prefix), 1e-12) : 1e-12;
}

// Oklab of reference XYZ / scale in FP64, stored as float (main.rs:1121-1130).
__global__ void __launch_bounds__(256) ref_lab_kernel(const double* __restrict__ ref_xyz, uint64_t samples,
                                                      const ScaleState* __restrict__ state,
                                                      float* __restrict__ ref_lab) {
    const uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= samples) return;
    const double scale = state->scale;
    const double x = ref_xyz[s * 3] / scale, y = ref_xyz[s * 3 + 1] / scale, z = ref_xyz[s * 3 + 2] / scale;
    const double l = cbrt(0.8189330101 * x + 0.3618667424 * y - 0.1288597137 * z);
    const double m = cbrt(0.0329845436 * x + 0.9293118715 * y + 0.0361456387 * z);
    const double t = cbrt(0.0482003018 * x + 0.2643662691 * y + 0.6338517070 * z);
    ref_lab[s * 3] = float(0.2104542553 * l + 0.7936177850 * m - 0.0040720468 * t);
    ref_lab[s * 3 + 1] = float(1.9779984951 * l - 2.4285922050 * m + 0.4505937099 * t);
    ref_lab[s * 3 + 2] = float(0.0259040371 * l + 0.7827717662 * m - 0.8086757660 * t);
}

}  // namespace

cudaError_t launch_reference_scale(const double* ref_xyz, uint64_t samples, ScaleState* state, uint32_t* hist,
                                   uint32_t sms, cudaStream_t stream) {
    const uint32_t blocks = uint32_t(std::min<uint64_t>((samples + 1023u) / 1024u, std::max(1u, 2u * sms)));
    const uint32_t width[6] = {11u, 11u, 11u, 11u, 10u, 10u};
    uint32_t shift = 64u;
    for (int pass = 0; pass < 6; ++pass) {
        shift -= width[pass];
        scale_select_kernel<<<blocks, 256, 0, stream>>>(ref_xyz, samples, shift, width[pass], pass == 0 ? 1u : 0u,
                                                        state, hist);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    scale_value_kernel<<<1, 1, 0, stream>>>(state);
    return cudaGetLastError();
}

cudaError_t launch_reference_lab(const double* ref_xyz, uint64_t samples, const ScaleState* state, float* ref_lab,
                                 cudaStream_t stream) {
    const uint64_t blocks = (samples + 255u) / 256u;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    ref_lab_kernel<<<dim3(uint32_t(blocks)), 256, 0, stream>>>(ref_xyz, samples, state, ref_lab);
    return cudaGetLastError();
}

cudaError_t launch_score(const ScoreLaunch& w, cudaStream_t stream) {
    // the first digit's histogram comes from the distances, the two below it from one reading each
    const uint32_t groups = (w.combos + kCombos - 1u) / kCombos;
    const uint64_t tiles = (w.samples + kTile - 1u) / kTile;
    const uint32_t across = uint32_t(std::min<uint64_t>(tiles, std::max(1u, 6u * w.sms / groups)));
    distance_kernel<<<dim3(across, groups), 256, 0, stream>>>(w.bands, w.samples, w.ref_lab, w.inv_scale,
                                                              w.combo_bands, w.combo_xyz, w.combos, w.channels,
                                                              w.dist, w.state, w.hist);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const uint32_t shift[3] = {21u, 10u, 0u}, width[3] = {11u, 11u, 10u};
    const uint32_t readers = uint32_t(  // five blocks of 40 KB a SM, in one wave
        std::min<uint64_t>(tiles, std::max(1u, 5u * w.sms / w.combos)));
    for (int pass = 0; pass < 3; ++pass) {
        if (pass > 0) {
            select_hist_kernel<<<dim3(readers, w.combos), 256, 0, stream>>>(w.dist, w.samples, w.state, shift[pass],
                                                                            width[pass], w.hist);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        select_pick_kernel<<<w.combos, 256, 0, stream>>>(w.state, pass == 0 ? 1u : 0u, width[pass], w.hist);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace sky
