// adjoint_wave.cu — the differentiable renderer's kernels over the stage queues
// (stage_queues.cuh): the primal of P = Q and the path-replay gradient with
// segment integrals (adjoint.cu holds the estimators' derivation, the ray loop
// that small launches, event counting and the null-collision estimator take, and
// the primal of distinct P and Q).
//
// The stages are the tracer's (trace_wave.cuh): track, vertex, continue, start,
// a warp running one of them on 32 paths.  A path of the gradient carries its
// chain's radiance and loss weight, and with each ray the majorant optical depth
// that the tracker summed.  The terms of a ray's segment integral are added when
// the ray's end is taken up by its next stage, those of the vertices where they
// are made; band gradients stay in the lane's registers while its band does, the
// Mie albedo's and g's for the whole kernel, and layer gradients go to the warp's
// copy in shared memory, from which the warp moves them to the FP64 outputs every
// kFlushBatches of its batches.
//
// What bounds it: instruction issue, as the tracer.  The ray loop runs all event
// code once per ray: 8 to 10 of 32 lanes active.  16.8 M chains (128x64, 32 bands,
// 64 spp): primal 3.79 -> 2.18 ms, gradient with the primal's chain radiance 4.05 ->
// 3.04 ms; 67 M chains (16 renders of 256x128, 4 bands, 32 spp): 19.4 -> 10.1 ms and
// 29.7 -> 20.2 ms.  The primal issues at 83 % with 24 lanes active; the gradient at
// 53 % with 17: its code is still more than the instruction caches hold ("no
// instruction" 2.9 cycles per issue), and its layer gradients are shared-memory
// atomics (short scoreboard 2.2).

#include <algorithm>

#include "adjoint_device.cuh"
#include "launch_limits.h"
#include "stage_queues.cuh"

namespace sky {
namespace {

using wave::align16;
using wave::as_f;
using wave::as_u;
using wave::kBatch;
using wave::kNothing;
using wave::kOutOfWork;
using wave::kQContinue;
using wave::kQNone;
using wave::kQStart;
using wave::kQTrack;
using wave::kQVertex;
using wave::kQueues;
using wave::Queues;
using wave::queue_slots;
using wave::StageQueues;
using wave::Taken;

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kNoBand = 0xffffffffu;

// How a ray ended (Path B.y), and the paths without one: see trace_wave.cuh.
enum : uint32_t { kHit = 1u, kMiss = 2u, kOver = 3u, kFresh = 4u };
enum : uint32_t { kFlagShadow = 1u << 8, kFlagGround = 1u << 9, kFlagTop = 1u << 10, kFlagReplay = 1u << 11 };

// Rays left to the track queue, and crossings left to the next step, as in the tracer.
constexpr uint32_t kPark = 14, kCrossing = 3;

// Batches of a warp between two moves of its layer-gradient copies to the FP64
// gradient, the block's warps in turn.  An FP32 copy's rounding error grows with the
// terms that it takes between them: a copy of the block's as many as a copy of one
// warp's, both fewer than a warp's copy in the ray loop takes of the smallest launch that
// comes here.  Largest error of 54.8 M chains, relative to the largest gradient, without
// the moves, with them and in the ray loop: 114 layers (one copy per block) 3.1e-4,
// 1.9e-7 and 1.5e-5; 100 layers (one per warp) 1.0e-5, 3.5e-7 and 8.8e-6.  (256 batches:
// 4.3e-7 and 1.5e-6, and at 300 layers 14.2 M chains still 3 times the ray loop's.)  The
// moves cost 16.8 M chains of 64 layers 1.3 %, 54.8 M of 1000 layers 4.7 %, the fit's 67 M,
// without a layer gradient, nothing.
constexpr uint32_t kFlushBatches = 64;

// A path in shared memory, rows of 16 bytes: A-F as the tracer's, then
//   G  the vertex: unscaled Rayleigh, Mie and ozone coefficients, layer
//   H  (gradient) majorant optical depth and start of the ray's current piece,
//      the chain's radiance
//   I  (gradient) loss weight; the random stream's position at the ray's start
enum : uint32_t { kA = 0u, kB = 1u, kC = 2u, kD = 3u, kE = 4u, kF = 5u, kG = 6u, kH = 7u, kI = 8u };
template <bool kGrad>
__host__ __device__ constexpr uint32_t path_rows() {
    return kGrad ? 9u : 7u;
}

__device__ __forceinline__ Rng path_rng(const float4& C, uint32_t dim) {
    Rng r;
    r.k0 = as_u(C.x);
    r.k1 = as_u(C.y);
    r.k2 = (as_u(C.z) & 255u) * 1664525u + 1013904223u;
    r.dim = dim;
    return r;
}

__device__ __forceinline__ uint32_t quotient(uint32_t a, uint32_t d, uint32_t reciprocal, uint32_t& rest) {
    uint32_t q = __umulhi(a, reciprocal);
    rest = a - q * d;
    if (rest >= d) {
        ++q;
        rest -= d;
    }
    return q;
}

// The sample index behind the sample's key (Rng::init: an odd multiplier, inverted mod 2^32).
__device__ __forceinline__ uint32_t sample_of(uint32_t k1, const DevLaunch& L) {
    constexpr uint32_t kInverse = 4276115653u;  // 1664525^-1 mod 2^32
    static_assert(1664525u * kInverse == 1u, "inverse of the stream's multiplier");
    return (((k1 - 1013904223u) * kInverse) ^ L.seed_hi) - L.sample_offset;
}

__device__ __forceinline__ MergedGrid adj_grid(const AdjCtx& A, uint32_t band) {
    const uint32_t L = A.S.layer_count;
    MergedGrid G;
    G.radius = A.G.radius + band * (L + 1u);
    G.maj = A.G.maj + band * (L + 1u);
    G.map = A.G.map + band * L;
    G.count = int(__ldg(A.G.count + band));
    return G;
}

// adj_track() from where the ray was left until at most `park` of the warp's
// rays are under way; returns how the lane's ray ended (0: not yet).
template <bool kGrad>
__device__ __forceinline__ uint32_t adj_track_batch(const AdjCtx& A, bool alive, const RayGeo& g, float t_max,
                                                    uint32_t band, Rng& rng, float4& B, uint32_t& meta,
                                                    float& tau_bar, float& t_piece, uint32_t park) {
    const DevScene& S = A.S;
    const MergedGrid G = adj_grid(A, band);
    const AdjSet Q = resolve(A.P, S.layer_count, band);
    int m = int((meta >> 16) & 0xfffu), dir = int(meta >> 28) - 1;
    float t = B.x, tau = B.y, t_seg = B.z;
    float maj = alive ? __ldg(G.maj + m) : 1.0f;
    uint32_t ended = 0u;
    for (uint32_t step = 0u; step < 4096u; ++step) {  // a ray crosses at most 2 x 1024 shells
        // one expression, contracted as adj_track() has it
        float next_t = 0.0f;
        if (alive) next_t = t + tau / maj;
        for (;;) {
            if (alive && !(next_t < t_seg)) {
                if (kGrad) tau_bar += (t_seg - t_piece) * maj;
                if (dir == 0) {
                    ended = kMiss;
                    alive = false;
                } else {
                    tau = fmaxf(tau - (t_seg - t) * maj, 0.0f);
                    t = t_seg;
                    if (kGrad) t_piece = t_seg;
                    m += dir;
                    t_seg = merged_crossing(G, g, m, t, t_max, dir);
                    maj = __ldg(G.maj + m);
                    next_t = t + tau / maj;
                }
            }
            if (uint32_t(__popc(__ballot_sync(kFull, alive && !(next_t < t_seg)))) <= kCrossing) break;
        }
        if (alive && next_t < t_seg) {
            t = next_t;
            const float accept = rng.next() * maj;
            const AdjMed mq = adj_med(Q, adj_base(S, band, altitude_at(g, t, S.ground_radius)));
            if (accept < mq.t) {
                if (kGrad) tau_bar += (t - t_piece) * maj;
                ended = kHit;
                alive = false;
            } else {
                tau = -__logf(fmaxf(1.0f - rng.next(), 0.0000001f));
            }
        }
        if (uint32_t(__popc(__ballot_sync(kFull, alive))) <= park) break;
    }
    B = make_float4(t, ended ? as_f(ended) : tau, t_seg, as_f(rng.dim));
    meta = (meta & 0xffffu) | (uint32_t(m) << 16) | (uint32_t(dir + 1) << 28);
    return ended;
}

// The sums of the Rayleigh and Mie terms of a phase value or pdf with their
// roundings written out, as the compiler contracts them in the ray loop: the two
// kernels' chains then agree to the last bit but for two in a thousand.
__device__ __forceinline__ float mixed(const AdjMed& m, float rayleigh, float mie) {
    const float r = __fmul_rn(m.R, rayleigh);
    return m.Ms > 0.0f ? __fmaf_rn(m.Ms, mie, r) : r;
}
// The HG table at a cosine: hg_value() and the terms of vertex_terms().
struct HgSlot {
    float p0, p1, d0, d1, t;
    __device__ __forceinline__ HgSlot(const AdjSet& X, uint32_t bins, float mu) {
        uint32_t i0, i1;
        hg_slot(bins, mu, i0, i1, t);
        p0 = __ldg(X.phase + i0);
        p1 = __ldg(X.phase + i1);
        d0 = __ldg(X.dphase + i0);
        d1 = __ldg(X.dphase + i1);
    }
    __device__ __forceinline__ float value() const { return fmaxf(fmaf(t, p1 - p0, p0), 0.0f); }
    __device__ __forceinline__ float slope() const { return fmaf(t, d1 - d0, d0); }
};

// vertex_terms() with the table's values at hand.
__device__ __forceinline__ void vertex_terms_at(AdjAcc& a, const AdjSet& X, const HgSlot& slot, const AdjBase& b,
                                                const AdjMed& m, float pr, float weight) {
    if (weight == 0.0f) return;
    const float pm = slot.value();
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
        a.gG = fmaf(w * m.Ms, slot.slope(), a.gG);
        a.gM = fmaf(w * X.omega * __ldg(p + 1), b.uM * pm, a.gM);
    }
}
// The coefficients at a vertex for its NEE terms and continuation.
__device__ __forceinline__ AdjMed vertex_med(const AdjSet& X, const AdjBase& b) {
    AdjMed m = adj_med(X, b);
    m.s = __fadd_rn(m.R, m.Ms);
    return m;
}

__device__ __forceinline__ float warp_add(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

template <int kPhase, bool kGrad, bool kBatchOfRenders, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, 2)
    adjoint_wave_kernel(const __grid_constant__ AdjCtx A, const __grid_constant__ AdjJobs J,
                        double* __restrict__ layer_grad, double* __restrict__ band_grad, uint32_t paths,
                        uint32_t used_paths, uint32_t copies, unsigned long long* __restrict__ work_counter,
                        uint32_t* __restrict__ status) {
    constexpr uint32_t kRows = path_rows<kGrad>();
    extern __shared__ __align__(16) unsigned char smem[];
    float4* const pool = reinterpret_cast<float4*>(smem);
    Queues* const Q = reinterpret_cast<Queues*>(pool + size_t(paths) * kRows);
    const StageQueues queues(Q, paths, used_paths);
    const DevScene& S = A.S;
    const uint32_t Lc = S.layer_count, bands = S.band_count, bins = S.phase_bins;
    const uint32_t nlayer = 3u * Lc + 2u;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float* const grads = reinterpret_cast<float*>(
        smem + align16(size_t(paths) * kRows * 16u + sizeof(Queues) + size_t(kQueues) * queue_slots(paths) * 2u));
    // two copies per warp (of its even and its odd lanes), one, or one per block
    const bool two = copies == 2u * kWarps;
    float* const sg = kGrad && copies ? grads + (two ? warp * 2u + (lane & 1u) : warp % copies) * nlayer : nullptr;
    float* const sb = grads + copies * nlayer;
    for (uint32_t i = threadIdx.x; i < used_paths; i += blockDim.x)
        pool[i * kRows + kB] = make_float4(0.0f, as_f(kFresh), 0.0f, 0.0f);
    if (kGrad)
        for (uint32_t i = threadIdx.x; i < copies * nlayer + kAdjBandParams * bands; i += blockDim.x) grads[i] = 0.0f;
    __syncthreads();
    AdjAcc acc{sg, Lc, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float acc_solar = 0.0f;         // the solar multiplier's gradient
    uint32_t acc_band = kNoBand;    // the band of acc's band gradients
    bool watchdog = false;
    uint32_t idle = 0u, turn = warp & 3u;

    for (uint32_t batch = 0u;;) {
        uint32_t stage, take, id;
        const Taken taken = queues.take<wave::kMaxIdlePolls, false>(lane, turn, idle, batch, 0u, status, stage, take, id);
        if (taken == kOutOfWork) break;
        if (taken == kNothing) continue;
        if (kGrad && copies && batch % kFlushBatches == warp * (kFlushBatches / uint32_t(kWarps))) {
            float* const own = grads + (two ? warp * 2u : warp % copies) * nlayer;
#pragma unroll 1
            for (uint32_t i = lane; i < nlayer; i += 32u) {
                double v = double(atomicExch(own + i, 0.0f));
                if (two) v += double(atomicExch(own + nlayer + i, 0.0f));
                if (v != 0.0) atomicAdd(layer_grad + i, v);
            }
        }
        const bool on = lane < take;
        float4* const P = pool + id * kRows;
        uint32_t next = kQNone;
        bool tracing = false, set_up = false;
        V3 ray_org = mk(0.0f, 0.0f, 0.0f), ray_dir = ray_org;
        float4 RA = make_float4(0.0f, 0.0f, 0.0f, 0.0f), B = RA, C = RA;
        float tau_bar = 0.0f, t_piece = 0.0f;
        uint32_t meta = 0u;
        Rng rng;
        rng.k0 = rng.k1 = rng.k2 = rng.dim = 0u;
        if (on) {
            B = P[kB];
            if (as_u(B.y) != kFresh) {
                RA = P[kA];
                C = P[kC];
                meta = as_u(C.z);
                rng = path_rng(C, as_u(B.w));
                if (kGrad) {
                    tau_bar = P[kH].x;
                    t_piece = P[kH].y;
                }
            }
        }
        uint32_t band = meta & 255u, job = kBatchOfRenders ? as_u(C.w) & 0xffffu : 0u, ls = as_u(C.w) >> 16;
        const uint32_t state = as_u(B.y);

        if (kGrad && stage != kQTrack) {
            if (on && state != kFresh && band != acc_band) {
                if (acc_band != kNoBand) {
                    float* bg = sb + acc_band * kAdjBandParams;
                    atomicAdd(bg, acc.gR);
                    atomicAdd(bg + 1, acc.gM);
                    atomicAdd(bg + 2, acc.gO);
                    atomicAdd(bg + 3, acc_solar);
                }
                acc.gR = acc.gM = acc.gO = acc_solar = 0.0f;
                acc_band = band;
            }
        }
        // the segment integral of the ray that ended: its weight, its end and its place in the random stream
        float seg_weight = 0.0f, seg_end = RA.w;
        uint32_t seg_dim = rng.dim;
        if (kGrad && stage != kQTrack && on && (meta & kFlagReplay) && !(meta & kFlagShadow) &&
            (state == kHit || state == kMiss)) {
            // an outgoing ray's, from its first random number
            const float4 I = P[kI];
            seg_weight = I.x * resolve(A.P, Lc, band).kS * (P[kH].z - P[kE].w);
            seg_dim = as_u(I.z);
            if (state == kHit) seg_end = B.x;
        }
        const uint32_t seg_band = band;

        if (stage == kQTrack) {
            tracing = on;
        } else if (stage == kQVertex) {
            if (on) {
                const DevLaunch& L = J.j[job].L;
                const float4 D = P[kD], E = P[kE];
                const AdjSet X = resolve(A.P, Lc, band);
                V3 org = mk(D.x, D.y, D.z);
                const V3 dir = mk(E.x, E.y, E.z);
                float thr = D.w;
                bool ground = (meta & kFlagGround) != 0u, alive = true;
                if (!(meta & kFlagShadow)) {  // a new vertex
                    ls = 0u;
                    ground = state != kHit;
                    if (!ground) {
                        const RayGeo g{RA.x, RA.y, RA.z};
                        org = madd(org, dir, B.x);
                        const AdjBase hb = adj_base(S, band, altitude_at(g, B.x, S.ground_radius));
                        const AdjMed mq = adj_med(X, hb);
                        if (mq.t > 0.0f && mq.s > 0.0f) thr *= fminf(fmaxf(mq.s / mq.t, 0.0f), 1.0f);
                        alive = mq.t > 0.0f && mq.s > 0.0f && !(thr <= 0.0f);
                        if (alive) P[kG] = make_float4(hb.uR, hb.uM, hb.uO, as_f(uint32_t(hb.layer)));
                    } else {
                        org = madd(org, dir, RA.w);
                    }
                    P[kD] = make_float4(org.x, org.y, org.z, thr);
                    reinterpret_cast<float*>(&P[kF])[2] = 0.0f;  // the vertex's NEE sum
                }
                if (!alive) {
                    reinterpret_cast<float*>(&P[kE])[3] = fmaxf(E.w, 0.0f);
                    reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                    next = kQStart;
                } else {
                    const uint32_t lights = L.direct_light_samples;
                    meta = band | (meta & kFlagReplay) | kFlagShadow | (ground ? uint32_t(kFlagGround) : 0u);
                    next = kQContinue;
                    B = make_float4(0.0f, as_f(kHit), 0.0f, 0.0f);  // no sun: as a shadow ray that collides
                    while (ls < lights) {
                        ++ls;
                        const AdjJob& JJ = J.j[job];
                        const V3 ldir = sample_sun_cone(JJ.sun, JJ.sun_t, JJ.sun_b, S.one_minus_cos_max, rng);
                        float mu = dot3(dir, ldir);
                        if (ground) {
                            mu = fmaxf(dot3(normalize_or_y(org), ldir), 0.0f);
                            if (!(mu > 0.0f)) continue;
                        }
                        ray_org = madd(org, ldir, kRayEpsilonKm);
                        ray_dir = ldir;
                        reinterpret_cast<float*>(&P[kF])[3] = mu;
                        set_up = true;
                        break;
                    }
                    B.w = as_f(rng.dim);
                    P[kB] = B;
                    reinterpret_cast<float*>(&P[kC])[2] = as_f(meta);
                    reinterpret_cast<float*>(&P[kC])[3] = as_f(job | (ls << 16));
                }
            }
        } else if (stage == kQContinue) {
            if (on) {
                const DevLaunch& L = J.j[job].L;
                const float4 D = P[kD], E = P[kE], F = P[kF];
                const AdjSet X = resolve(A.P, Lc, band);
                const bool ground = (meta & kFlagGround) != 0u, replay = kGrad && (meta & kFlagReplay) != 0u;
                V3 org = mk(D.x, D.y, D.z), dir = mk(E.x, E.y, E.z);
                float nee = F.z;
                AdjBase hb{0.0f, 0.0f, 0.0f, 0};
                if (!ground) {
                    const float4 G = P[kG];
                    hb = AdjBase{G.x, G.y, G.z, int(as_u(G.w))};
                }
                const AdjMed mq = vertex_med(X, hb);
                const uint32_t lights = L.direct_light_samples;
                const bool lit = state == kMiss, more_lights = ls < lights;
                const float w = kGrad ? P[kI].x * X.kS : 0.0f;
                float thr = D.w, rad = E.w;
                V3 nd = mk(0.0f, 1.0f, 0.0f), axis = dir;
                float cos_t = 1.0f, sin_t = 0.0f, xi_phi = 0.0f;
                bool framed = true;
                if (lit && ground) {
                    const float term =
                        S.ground_albedo * kInvPi * __ldg(&S.bands[band].solar_radiance) * F.w / S.light_pdf;
                    nee = __fadd_rn(nee, term);
                    if (kGrad) seg_weight = w * thr * term * (1.0f / float(lights));
                }
                // the phase function at a medium vertex, once for the lit sun sample's term (its
                // transmittance is 1, sky_trace.wgsl:566-608) and once for the continuation,
                // by the same code (one copy of it in the gradient, whose code is large: 3.44 ->
                // 3.09 ms; two in the primal, where one is 5 % slower)
                constexpr int kCopies = kGrad ? 1 : 2;
#pragma unroll kCopies
                for (uint32_t k = 0u; k < 2u; ++k) {
                    float mu = F.w, pdf = 1.0f;
                    if (k == 0u) {
                        if (ground || !lit) continue;
                    } else {
                        if (more_lights) break;
                        rad += thr * (nee * (1.0f / float(lights)));
                        if (ground) break;
                        if (kPhase == SKY_PHASE_TABULATED) {
                            const float target = rng.next() * mq.s;
                            const bool rayleigh = target < mq.R || !(mq.Ms > 0.0f);
                            const float xi_mu = rng.next();
                            mu = rayleigh ? invert_rayleigh_cdf(xi_mu) : hg_sample_mu(X, bins, xi_mu);
                            xi_phi = rng.next();
                            cos_t = fminf(fmaxf(mu, -1.0f), 1.0f);
                            sin_t = sqrtf(fmaxf(1.0f - cos_t * cos_t, 0.0f));
                            pdf = mixed(mq, rayleigh_phase(mu), mq.Ms > 0.0f ? hg_sampling_pdf(X, bins, mu) : 0.0f);
                        } else {
                            nd = sample_isotropic(rng);
                            framed = false;
                            mu = dot3(dir, nd);
                        }
                    }
                    const HgSlot slot(X, bins, mu);
                    const float pr = rayleigh_phase(mu), pm = mq.Ms > 0.0f ? slot.value() : 0.0f;
                    float weight;
                    if (k == 0u) {
                        const float sum = __fadd_rn(__fmul_rn(mq.R, pr), mq.Ms > 0.0f ? __fmul_rn(mq.Ms, pm) : 0.0f);
                        const float ph = mq.s > 0.0f ? sum / mq.s : 0.0f;
                        const float term = __ldg(&S.bands[band].solar_radiance) * ph / S.light_pdf;
                        nee = __fadd_rn(nee, term);  // not contracted into the term's division
                        weight = kGrad ? w * thr * term * (1.0f / float(lights)) : 0.0f;
                        if (kGrad) seg_weight = weight;
                    } else {
                        const float value = mixed(mq, pr, pm);
                        thr *= kPhase == SKY_PHASE_TABULATED ? value / pdf : value / mq.s / kIsotropicPdf;
                        weight = kGrad ? w * (P[kH].z - rad) : 0.0f;
                    }
                    if (replay) vertex_terms_at(acc, X, slot, hb, mq, pr, weight);
                }
                if (kGrad && !replay) seg_weight = 0.0f;
                if (more_lights) {
                    reinterpret_cast<float*>(&P[kF])[2] = nee;
                    next = kQVertex;
                } else {
                    uint32_t depth = as_u(F.x);
                    // each branch has drawn its angles; one shared frame step turns them into
                    // the direction (as direction_from_axis_mu / sample_cosine_hemisphere)
                    if (ground) {
                        // the Lambert bounce (sky_trace.wgsl:750-766)
                        axis = normalize_or_y(org);
                        const float u = rng.next();
                        sin_t = sqrtf(u);
                        xi_phi = rng.next();
                        cos_t = sqrtf(fmaxf(1.0f - u, 0.0f));
                    }
                    V3 fn = axis;
                    if (framed) {
                        V3 t, bt;
                        orthonormal_basis(axis, t, bt);
                        fn = normalize_or_y(axis);
                        nd = direction_from_frame(fn, t, bt, cos_t, sin_t, xi_phi);
                    }
                    bool alive = true;
                    if (ground) {
                        const float pdf = fmaxf(dot3(fn, nd), 0.0f) * kInvPi;
                        const float cos_out = fmaxf(dot3(axis, nd), 0.0f);
                        if (pdf <= 0.0f || cos_out <= 0.0f) {
                            alive = false;
                        } else {
                            const float f = S.ground_albedo * kInvPi * cos_out / pdf;
                            thr *= f;
                        }
                    }
                    if (alive && depth >= L.rr_start_depth) {  // russian_roulette (sky_trace.wgsl:691-701)
                        const float q = fminf(fmaxf(thr, 0.05f), 0.95f);
                        if (rng.next() > q) alive = false;
                        else thr = thr / q;
                    }
                    if (!alive) {
                        rad = fmaxf(rad, 0.0f);
                    } else {
                        org = madd(org, nd, kRayEpsilonKm);
                        dir = nd;
                        if (rad < 0.0f || rad != rad || thr < 0.0f || thr != thr) {
                            rad = 0.0f;
                            alive = false;
                        } else if (++depth >= L.watchdog_limit) {
                            watchdog = true;
                            alive = false;
                        }
                    }
                    P[kD] = make_float4(org.x, org.y, org.z, thr);
                    P[kE] = make_float4(dir.x, dir.y, dir.z, rad);
                    reinterpret_cast<float*>(&P[kF])[0] = as_f(depth);
                    set_up = alive;
                    ray_org = org;
                    ray_dir = dir;
                    meta = band | (meta & kFlagReplay);
                    if (!alive) {
                        reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                        next = kQStart;
                    }
                }
            }
        } else {
            // the chains that ended: a gradient's first trace goes over into its replay
            bool again = false;
            if (on && state != kFresh) {
                const AdjJob& JJ = J.j[job];
                const float4 E = P[kE], F = P[kF];
                const uint32_t cell = as_u(F.y);
                float rad = E.w;
                if (state == kMiss) {  // left through the top of the atmosphere
                    if (as_u(F.x) == 0u && dot3(mk(E.x, E.y, E.z), load3(JJ.sun)) >= S.cos_max)
                        rad += P[kD].w * __ldg(&S.bands[band].solar_radiance);
                    rad = fmaxf(rad, 0.0f);
                }
                if (!kGrad) {
                    if (JJ.chain_rad) JJ.chain_rad[uint64_t(cell) * JJ.L.spp + sample_of(as_u(C.y), JJ.L)] = rad;
                    if (rad != 0.0f) {  // the sums start at zero, or hold what they are added to
                        const double rd = double(resolve(A.P, Lc, band).kS * rad);
                        atomicAdd(JJ.cell_sum + cell, rd);
                        if (JJ.cell_sumsq) atomicAdd(JJ.cell_sumsq + cell, rd * rd);
                    }
                } else if (!(meta & kFlagReplay)) {
                    again = rad > 0.0f;
                    if (again) reinterpret_cast<float*>(&P[kH])[2] = rad;
                    else if (rad != 0.0f) acc_solar = fmaf(P[kI].x, rad, acc_solar);
                } else {
                    acc_solar = fmaf(P[kI].x, P[kH].z, acc_solar);
                }
            }
            // the next samples of the launch, band-major within a render (trace_wave.cuh)
            const uint32_t wanted = __ballot_sync(kFull, on && !again);
            unsigned long long base = 0u;
            if (lane == 0u && wanted) base = atomicAdd(work_counter, (unsigned long long)__popc(wanted));
            base = __shfl_sync(kFull, base, 0);
            const unsigned long long at = base + __popc(wanted & ((1u << lane) - 1u));
            const bool more = on && !again && at < J.chains;
            uint32_t slab_pixel = 0u, k1 = as_u(C.y);
            bool start = again;
            if (again) {
                slab_pixel = as_u(P[kF].y) / bands;
            } else if (more) {
                job = 0u;
                if constexpr (kBatchOfRenders) {
                    uint32_t hi = J.count;
                    while (hi - job > 1u) {
                        const uint32_t mid = (job + hi) >> 1;
                        if (J.j[mid].chain_begin <= at) job = mid;
                        else hi = mid;
                    }
                }
                const AdjJob& JJ = J.j[job];
                const DevLaunch& L = JJ.L;
                const unsigned long long rel = at - JJ.chain_begin;
                uint32_t c = uint32_t(__umul64hi(rel, L.spp_reciprocal));
                uint32_t sample = uint32_t(rel - (unsigned long long)c * L.spp);
                if (sample >= L.spp) {
                    ++c;
                    sample -= L.spp;
                }
                band = quotient(c, L.width * L.rows, L.pixels_reciprocal, slab_pixel);
                const uint32_t cell = slab_pixel * bands + band;
                k1 = ((L.sample_offset + sample) ^ L.seed_hi) * 1664525u + 1013904223u;
                meta = band;
                start = true;
                if (kGrad) {
                    const float dloss = __ldg(JJ.dloss + cell), wc = dloss * (1.0f / float(L.spp));
                    float total = 0.0f;
                    if (dloss == 0.0f) {
                        start = false;  // no loss: no gradient
                    } else if (JJ.chain_rad) {
                        // the forward's radiance of this chain stands in for its first trace
                        total = __ldg(JJ.chain_rad + uint64_t(cell) * L.spp + sample);
                        meta |= kFlagReplay;
                        if (!(total > 0.0f)) {
                            if (total != 0.0f) atomicAdd(sb + band * kAdjBandParams + 3u, wc * total);
                            start = false;
                        }
                    }
                    P[kH] = make_float4(0.0f, 0.0f, total, 0.0f);
                    P[kI] = make_float4(wc, 0.0f, 0.0f, 0.0f);
                }
                P[kF] = make_float4(as_f(0u), as_f(cell), 0.0f, 0.0f);
                if (!start) {  // nothing to trace: as a path without a chain
                    reinterpret_cast<float*>(&P[kB])[1] = as_f(kFresh);
                    next = kQStart;
                }
            }
            const uint32_t gone = __popc(__ballot_sync(kFull, on && !again && !more));
            if (gone && lane == 0u) atomicSub(&Q->live, gone);
            if (start) {
                const DevLaunch& L = J.j[job].L;
                uint32_t px;
                const uint32_t py = quotient(slab_pixel, L.width, L.width_reciprocal, px) + L.row_begin;
                rng.init(py * L.width + px, 0u, band, L.seed_lo, L.seed_hi);
                rng.k1 = k1;
                if (again) {
                    meta = band | kFlagReplay;
                    reinterpret_cast<float*>(&P[kF])[0] = as_f(0u);
                }
                const V3 dir = camera_dir(L, px, py, rng);
                const V3 org = mk(0.0f, S.ground_radius + fmaxf(L.observer_altitude, 0.0f), 0.0f);
                set_up = true;
                ray_org = org;
                ray_dir = dir;
                P[kC] = make_float4(as_f(rng.k0), as_f(rng.k1), as_f(meta), as_f(job));
                P[kD] = make_float4(org.x, org.y, org.z, 1.0f);
                P[kE] = make_float4(dir.x, dir.y, dir.z, 0.0f);
            }
        }

        if (kGrad && seg_weight != 0.0f) {
            Rng at = rng;
            at.dim = seg_dim;
            at.k0 = as_u(C.x);
            at.k1 = as_u(C.y);
            at.k2 = seg_band * 1664525u + 1013904223u;
            const RayGeo g{RA.x, RA.y, RA.z};
            segment_terms(A, resolve(A.P, Lc, seg_band), seg_band, g, seg_end, tau_bar, seg_weight, at, acc);
        }
        // the stages' rays, as the tracer sets them up
        if (set_up) {
            const RayGeo g = ray_geo(ray_org, ray_dir);
            const uint32_t word = as_u(reinterpret_cast<const float*>(&P[kC])[3]);
            const DevLaunch& L = J.j[kBatchOfRenders ? word & 0xffffu : 0u].L;
            float t_max;
            uint32_t boundary;
            bool ok = next_boundary(S, g, t_max, boundary);
            if (meta & kFlagShadow) {
                ok = ok && boundary == 1u;
                if (!ok && (word >> 16) < L.direct_light_samples) next = kQVertex;  // the next sample
            } else {
                if (L.max_orders != 0u && as_u(reinterpret_cast<const float*>(&P[kF])[0]) >= L.max_orders) ok = false;
                if (boundary == 1u) meta |= kFlagTop;
                if (!ok) {
                    float* rad = reinterpret_cast<float*>(&P[kE]) + 3;
                    *rad = fmaxf(*rad, 0.0f);
                    reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                    reinterpret_cast<float*>(&P[kC])[2] = as_f(meta);
                    next = kQStart;
                }
            }
            if (ok) {
                if (kGrad) reinterpret_cast<float*>(&P[kI])[2] = as_f(rng.dim);
                const MergedGrid G = adj_grid(A, band);
                const int m = merged_layer_at(S, G, altitude_at(g, fminf(kRayEpsilonKm, t_max), S.ground_radius));
                int dir;
                const float t_seg = merged_crossing(G, g, m, 0.0f, t_max, dir);
                const float tau = -__logf(fmaxf(1.0f - rng.next(), 0.0000001f));
                B = make_float4(0.0f, tau, t_seg, as_f(rng.dim));
                meta = (meta & 0xffffu) | (uint32_t(m) << 16) | (uint32_t(dir + 1) << 28);
                RA = make_float4(g.b, g.p, g.r0sq, t_max);
                tau_bar = t_piece = 0.0f;
                tracing = true;
            }
        }
        const uint32_t rays = __popc(__ballot_sync(kFull, tracing));
        if (rays) {
            const RayGeo g{RA.x, RA.y, RA.z};
            const uint32_t ended = adj_track_batch<kGrad>(A, tracing, g, RA.w, band, rng, B, meta, tau_bar, t_piece,
                                                          min(kPark, rays / 2u));
            if (tracing) {
                if (!ended) next = kQTrack;
                else if (meta & kFlagShadow) next = kQContinue;
                else next = ended == kMiss && (meta & kFlagTop) ? kQStart : kQVertex;
                if (kGrad || next == kQTrack || next == kQVertex) P[kA] = RA;
                P[kB] = B;
                reinterpret_cast<float*>(&P[kC])[2] = as_f(meta);
                if (kGrad) {
                    reinterpret_cast<float*>(&P[kH])[0] = tau_bar;
                    reinterpret_cast<float*>(&P[kH])[1] = t_piece;
                }
            }
        }
        queues.put(lane, next, id, status);
    }
    if (__any_sync(kFull, watchdog) && lane == 0u) atomicOr(status, 1u);
    if (!kGrad) return;
    // the lanes' sums: one addition per warp where its lanes hold the same band
    const float gw = warp_add(acc.gW), gg = warp_add(acc.gG);
    const uint32_t one = __shfl_sync(kFull, acc_band, 0);
    if (__all_sync(kFull, acc_band == one)) {
        const float v0 = warp_add(acc.gR), v1 = warp_add(acc.gM), v2 = warp_add(acc.gO), v3 = warp_add(acc_solar);
        acc.gR = lane == 0u ? v0 : 0.0f;
        acc.gM = lane == 0u ? v1 : 0.0f;
        acc.gO = lane == 0u ? v2 : 0.0f;
        acc_solar = lane == 0u ? v3 : 0.0f;
    }
    if (acc_band != kNoBand && (acc.gR != 0.0f || acc.gM != 0.0f || acc.gO != 0.0f || acc_solar != 0.0f)) {
        float* bg = sb + acc_band * kAdjBandParams;
        atomicAdd(bg, acc.gR);
        atomicAdd(bg + 1, acc.gM);
        atomicAdd(bg + 2, acc.gO);
        atomicAdd(bg + 3, acc_solar);
    }
    if (lane == 0u && sg) {
        atomicAdd(sg + 3u * Lc, gw);
        atomicAdd(sg + 3u * Lc + 1u, gg);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; layer_grad && i < nlayer; i += blockDim.x) {
        double v = 0.0;
        for (uint32_t k = 0; k < copies; ++k) v += double(grads[k * nlayer + i]);
        if (v != 0.0) atomicAdd(layer_grad + i, v);
    }
    if (band_grad)
        for (uint32_t i = threadIdx.x; i < kAdjBandParams * bands; i += blockDim.x)
            if (sb[i] != 0.0f) atomicAdd(band_grad + i, double(sb[i]));
}

template <int kPhase, bool kGrad, bool kBatchOfRenders>
cudaError_t launch_shape(const AdjCtx& A, const AdjJobs& J, double* layer_grad, double* band_grad, uint32_t* status,
                         unsigned long long* work_counter, cudaStream_t stream) {
    constexpr int kWarps = kGrad ? 12 : 16;  // 80 and 64 registers per lane
    constexpr uint32_t kThreads = kWarps * 32u;
    const void* k = reinterpret_cast<const void*>(adjoint_wave_kernel<kPhase, kGrad, kBatchOfRenders, kWarps>);
    int dev = 0, sms = 0, per_sm = 0, smem_sm = 0, smem_block = 0, reserved = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&smem_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
        return e;
    // two layer-gradient copies per warp, of its even and its odd lanes (an FP32 addition in shared
    // memory is repeated for each lane that meets another at its address; 16.8 M chains, 64 layers: one
    // 3.09, two 3.00, four 2.98 ms), while two blocks of them leave the paths room; else one per
    // warp, or one
    const size_t nlayer = 3u * A.S.layer_count + 2u, nband = kGrad ? size_t(kAdjBandParams) * A.S.band_count : 0u;
    const size_t warp_copy = kWarps * nlayer * sizeof(float);
    const uint32_t copies = !kGrad || !layer_grad         ? 0u
                            : warp_copy <= 12u * 1024u ? 2u * uint32_t(kWarps)
                            : warp_copy <= 16u * 1024u ? uint32_t(kWarps)
                                                       : 1u;
    const size_t extra = (copies * nlayer + nband) * sizeof(float);
    auto bytes = [&](uint32_t p) {
        return align16(size_t(p) * path_rows<kGrad>() * 16u + sizeof(Queues) +
                       size_t(kQueues) * queue_slots(p) * sizeof(uint16_t)) + extra;
    };
    auto fits = [&](uint32_t p, int blocks) {
        return bytes(p) <= size_t(smem_block) && size_t(blocks) * (bytes(p) + size_t(reserved)) <= size_t(smem_sm);
    };
    uint32_t paths = kThreads * 5u / 4u;
    while (paths > kThreads && !fits(paths, 2)) paths -= 32u;
    if (!fits(paths, 2)) {
        paths = kThreads * 5u / 4u;
        while (paths > 32u && !fits(paths, 1)) paths -= 32u;
    }
    const size_t smem = bytes(paths);
    if ((e = allow_shared_memory(k, smem)) != cudaSuccess) return e;
    const size_t need = size_t(fits(paths, 2) ? 2 : 1) * (smem + size_t(reserved));
    const int pct = int(std::min<size_t>(100u, (need * 100u + size_t(smem_sm) - 1u) / size_t(smem_sm)));
    if (cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, std::max(pct, 1)) != cudaSuccess)
        (void)cudaGetLastError();  // a hint
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem)) != cudaSuccess) return e;
    const uint64_t want = (J.chains + 31u) / 32u;
    const uint32_t blocks = uint32_t(std::max<uint64_t>(1u, std::min<uint64_t>(uint64_t(std::max(per_sm, 1)) * sms, want)));
    const uint32_t used = uint32_t(std::min<uint64_t>(paths, ((J.chains + blocks - 1u) / blocks + 31u) / 32u * 32u));
    adjoint_wave_kernel<kPhase, kGrad, kBatchOfRenders, kWarps><<<blocks, kThreads, smem, stream>>>(
        A, J, layer_grad, band_grad, paths, used, copies, work_counter, status);
    return cudaGetLastError();
}

template <int kPhase, bool kGrad>
cudaError_t launch_count(const AdjCtx& A, const AdjJobs& J, double* layer_grad, double* band_grad, uint32_t* status,
                         unsigned long long* work_counter, cudaStream_t stream) {
    return J.count > 1u ? launch_shape<kPhase, kGrad, true>(A, J, layer_grad, band_grad, status, work_counter, stream)
                        : launch_shape<kPhase, kGrad, false>(A, J, layer_grad, band_grad, status, work_counter, stream);
}

}  // namespace

// Few chains per lane of the chip (1024 lanes per SM): the ray loop of adjoint.cu.
// Measured with both (ms, ray loop against queues): primal 1.0 M chains 0.52 / 0.55,
// 2.1 M 0.70 / 0.66: 10 per lane; gradient 4.7 M 1.27 / 1.35, 8.4 M 2.11 / 2.00: 44.
cudaError_t adjoint_small(const AdjJobs& J, bool grad, bool& small) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    small = J.chains < (grad ? 44u : 10u) * 1024u * uint64_t(sms);
    return e;
}

cudaError_t launch_adjoint_wave(const AdjCtx& A, const AdjJobs& J, bool grad, double* layer_grad, double* band_grad,
                                uint32_t* status, unsigned long long* work_counter, cudaStream_t stream) {
    const bool tabulated = J.j[0].L.phase_sampling == SKY_PHASE_TABULATED;
    if (grad)
        return tabulated
                   ? launch_count<SKY_PHASE_TABULATED, true>(A, J, layer_grad, band_grad, status, work_counter, stream)
                   : launch_count<SKY_PHASE_ISOTROPIC, true>(A, J, layer_grad, band_grad, status, work_counter, stream);
    return tabulated
               ? launch_count<SKY_PHASE_TABULATED, false>(A, J, nullptr, nullptr, status, work_counter, stream)
               : launch_count<SKY_PHASE_ISOTROPIC, false>(A, J, nullptr, nullptr, status, work_counter, stream);
}

}  // namespace sky
