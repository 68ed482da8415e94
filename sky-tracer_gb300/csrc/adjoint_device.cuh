// adjoint_device.cuh — device functions of the differentiable renderer's kernels
// (adjoint.cu, adjoint_wave.cu): the parameterised medium, its phase function
// and the gradient terms.

#pragma once

#include "adjoint_kernels.h"
#include "sky_device.cuh"

namespace sky {
namespace {

// Unscaled coefficients at a point: air xs_R, m0 ext0 and o3 xs_O of the
// band, and the uniform layer that holds the point.
struct AdjBase {
    float uR, uM, uO;
    int layer;
};

// Coefficients of one parameter set at a point.
struct AdjMed {
    float R, M, O, Ms, t, s;
};

// A parameter set resolved for one band.
struct AdjSet {
    const float* layer;
    float kR, kM, kO, kS;
    float omega;
    const float* phase;
    const float* dphase;
    const float* cdf;
    const float* bin_pdf;
};

__device__ __forceinline__ AdjSet resolve(const AdjParamSet& X, uint32_t layers, uint32_t band) {
    AdjSet r;
    r.layer = X.layer;
    if (X.band) {
        const float* k = X.band + band * kAdjBandParams;
        r.kR = __ldg(k);
        r.kM = __ldg(k + 1);
        r.kO = __ldg(k + 2);
        r.kS = __ldg(k + 3);
    } else {
        r.kR = r.kM = r.kO = r.kS = 1.0f;
    }
    r.omega = __ldg(X.layer + 3 * layers);
    r.phase = X.phase;
    r.dphase = X.dphase;
    r.cdf = X.cdf;
    r.bin_pdf = X.bin_pdf;
    return r;
}

__device__ __forceinline__ AdjBase adj_base(const DevScene& S, uint32_t band, float alt) {
    AdjBase b;
    b.uR = b.uM = b.uO = 0.0f;
    b.layer = 0;
    if (!(alt >= 0.0f && alt <= S.top_altitude)) return b;
    const uint32_t k = knot_interval(S, S.knot_z, S.finder, alt);
    const float dz = alt - S.knot_z[k];
    const DevProfileKnot& P = S.profile[k];
    const DevBand& B = S.bands[band];
    b.uR = fmaxf(fmaf(dz, P.air_slope, P.air) * B.rayleigh_xs, 0.0f);
    b.uO = fmaxf(fmaf(dz, P.ozone_slope, P.ozone) * B.ozone_xs, 0.0f);
    const float mass = fmaxf(fmaf(dz, P.mass_slope[0], P.mass[0]), 0.0f);
    const SkyAerosolOptics o = S.optics[band * kSpecies];
    b.uM = fmaxf(mass * o.scattering_km_inv_per_g_m3, 0.0f) + fmaxf(mass * o.absorption_km_inv_per_g_m3, 0.0f);
    b.layer = min(int(alt * S.inv_layer_dz), int(S.layer_count) - 1);
    return b;
}

__device__ __forceinline__ AdjMed adj_med(const AdjSet& X, const AdjBase& b) {
    const float* p = X.layer + 3 * b.layer;
    AdjMed m;
    m.R = __ldg(p) * X.kR * b.uR;
    m.M = __ldg(p + 1) * X.kM * b.uM;
    m.O = __ldg(p + 2) * X.kO * b.uO;
    m.Ms = X.omega * m.M;
    m.s = m.R + m.Ms;
    m.t = m.R + m.M + m.O;
    return m;
}

// Position of mu on the cube-root grid (mie_phase, sky_trace.wgsl:485-494).
__device__ __forceinline__ void hg_slot(uint32_t bins, float mu, uint32_t& i0, uint32_t& i1, float& t) {
    const float u = cbrt_pos((1.0f - fminf(fmaxf(mu, -1.0f), 1.0f)) * 0.5f);
    const float f = u * float(bins) - 0.5f;
    i0 = min(uint32_t(fminf(fmaxf(floorf(f), 0.0f), float(bins - 1u))), bins - 1u);
    i1 = min(i0 + 1u, bins - 1u);
    t = fminf(fmaxf(f - float(i0), 0.0f), 1.0f);
}

__device__ __forceinline__ float hg_value(const AdjSet& X, uint32_t bins, float mu) {
    uint32_t i0, i1;
    float t;
    hg_slot(bins, mu, i0, i1, t);
    const float p0 = __ldg(X.phase + i0), p1 = __ldg(X.phase + i1);
    return fmaxf(fmaf(t, p1 - p0, p0), 0.0f);
}

// sum_i sigma_i p_i(mu): the scattering-vertex factor.
__device__ __forceinline__ float vertex_phase(const AdjSet& X, uint32_t bins, const AdjMed& m, float mu) {
    return m.R * rayleigh_phase(mu) + (m.Ms > 0.0f ? m.Ms * hg_value(X, bins, mu) : 0.0f);
}

// Gradient accumulator of one lane: per-layer scales in the warp's copy of
// the layer gradient in shared memory; the Mie albedo and g, and the
// multipliers of the lane's band, in registers.
struct AdjAcc {
    float* sg;  // [3 L + 2]
    uint32_t L;
    float gR, gM, gO;  // band multipliers
    float gW, gG;      // Mie albedo, Mie g
};

// d sigma_t terms of a null collision, times c (= -weight / sigma_n).
__device__ __forceinline__ void null_terms(AdjAcc& a, const AdjSet& X, const AdjBase& b, float c) {
    const float* p = X.layer + 3 * b.layer;
    float* g = a.sg ? a.sg + 3 * b.layer : nullptr;  // null: band gradients only
    if (b.uR > 0.0f) {
        if (g) atomicAdd(g, c * X.kR * b.uR);
        a.gR = fmaf(c * __ldg(p), b.uR, a.gR);
    }
    if (b.uM > 0.0f) {
        if (g) atomicAdd(g + 1, c * X.kM * b.uM);
        a.gM = fmaf(c * __ldg(p + 1), b.uM, a.gM);
    }
    if (b.uO > 0.0f) {
        if (g) atomicAdd(g + 2, c * X.kO * b.uO);
        a.gO = fmaf(c * __ldg(p + 2), b.uO, a.gO);
    }
}

// weight * d log(sum_i sigma_i p_i(mu)) of a scattering vertex.
__device__ __forceinline__ void vertex_terms(AdjAcc& a, const AdjSet& X, uint32_t bins, const AdjBase& b,
                                             const AdjMed& m, float mu, float weight) {
    if (weight == 0.0f) return;
    uint32_t i0, i1;
    float t;
    hg_slot(bins, mu, i0, i1, t);
    const float p0 = __ldg(X.phase + i0), p1 = __ldg(X.phase + i1);
    const float pm = fmaxf(fmaf(t, p1 - p0, p0), 0.0f);
    const float d0 = __ldg(X.dphase + i0), d1 = __ldg(X.dphase + i1);
    const float dpm = fmaf(t, d1 - d0, d0);
    const float pr = rayleigh_phase(mu);
    const float sum = m.R * pr + m.Ms * pm;
    if (!(sum > 0.0f)) return;
    const float w = weight / sum;
    const float* p = X.layer + 3 * b.layer;
    float* g = a.sg ? a.sg + 3 * b.layer : nullptr;
    if (b.uR > 0.0f) {
        if (g) atomicAdd(g, w * X.kR * b.uR * pr);
        a.gR = fmaf(w * __ldg(p), b.uR * pr, a.gR);
    }
    if (b.uM > 0.0f) {
        if (g) atomicAdd(g + 1, w * X.omega * X.kM * b.uM * pm);
        a.gW = fmaf(w * m.M, pm, a.gW);
        a.gG = fmaf(w * m.Ms, dpm, a.gG);
        a.gM = fmaf(w * X.omega * __ldg(p + 1), b.uM * pm, a.gM);
    }
}

// Estimate of -integral d(sigma_t) over [0, t_end] of a ray, times weight:
// N points stratified in the majorant optical depth of Q's tracking grid
// (density mu_bar / tau_bar along the ray; tau_bar as the tracker summed
// it), each adding -weight (tau_bar / N) d(sigma_t) / mu_bar.  N grows with
// tau_bar.  The
// points' random numbers come from a stream of their own (another pcg4d
// key, 16 draws per position of the path's stream), so the path's own
// draws are untouched.
constexpr int kMaxSegmentPoints = 4;

__device__ __forceinline__ void segment_terms(const AdjCtx& A, const AdjSet& Q, uint32_t band, const RayGeo& g,
                                              float t_end, float tau, float weight, const Rng& rng, AdjAcc& acc) {
    if (weight == 0.0f || !(t_end > 0.0f) || !(tau > 0.0f)) return;
    const DevScene& S = A.S;
    const uint32_t L = S.layer_count;
    MergedGrid G;
    G.radius = A.G.radius + band * (L + 1u);
    G.maj = A.G.maj + band * (L + 1u);
    G.map = A.G.map + band * L;
    G.count = int(__ldg(A.G.count + band));
    const int m0 = merged_layer_at(S, G, altitude_at(g, fminf(kRayEpsilonKm, t_end), S.ground_radius));
    const int guard_max = 2 * G.count + 4;
    float t = 0.0f;
    int m = m0, dir = 0;
    const int n = min(kMaxSegmentPoints, 1 + int(tau));
    const float step = tau / float(n);
    Rng r2 = rng;  // 16 draws of its own per position of the path's stream
    r2.k2 ^= 0x68E31DA4u;
    r2.dim = rng.dim * 16u;
    int j = 0;
    float uj = r2.next() * step;
    float u0 = 0.0f;
    t = 0.0f;
    m = m0;
    for (int guard = 0; guard < guard_max && j < n; ++guard) {
        const float t_seg = merged_crossing(G, g, m, t, t_end, dir);
        const float maj = __ldg(G.maj + m);
        const float u1 = u0 + (t_seg - t) * maj;
        while (j < n && (uj < u1 || dir == 0)) {
            const float tj = fminf(t + (uj - u0) / maj, t_seg);
            const AdjBase b = adj_base(S, band, altitude_at(g, tj, S.ground_radius));
            null_terms(acc, Q, b, -weight * step / maj);
            ++j;
            uj = (float(j) + r2.next()) * step;
        }
        if (dir == 0) break;
        u0 = u1;
        t = t_seg;
        m += dir;
    }
}

// Inverse CDF of an HG table (MiePhaseTable::sample_mu_pdf, phase.rs:53-69).
__device__ __forceinline__ float hg_sample_mu(const AdjSet& X, uint32_t bins, float xi) {
    xi = fminf(fmaxf(xi, 0.0f), 1.0f - kF32Epsilon);
    uint32_t lo = 0, hi = bins;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(X.cdf + mid) <= xi) lo = mid + 1u;
        else hi = mid;
    }
    const uint32_t bin = min(lo, bins - 1u);
    const float prev = bin == 0u ? 0.0f : __ldg(X.cdf + bin - 1u);
    const float next = __ldg(X.cdf + bin);
    const float t = next > prev ? (xi - prev) / (next - prev) : 0.5f;
    return mu_edge(bin, bins) * (1.0f - t) + mu_edge(bin + 1u, bins) * t;
}

// MiePhaseTable::sampling_pdf (phase.rs:71-75)
__device__ __forceinline__ float hg_sampling_pdf(const AdjSet& X, uint32_t bins, float mu) {
    const float u = cbrt_pos((1.0f - fminf(fmaxf(mu, -1.0f), 1.0f)) * 0.5f);
    const uint32_t bin = min(uint32_t(floorf(u * float(bins))), bins - 1u);
    return fmaxf(__ldg(X.bin_pdf + bin), 1.0e-12f);
}

}  // namespace
}  // namespace sky
