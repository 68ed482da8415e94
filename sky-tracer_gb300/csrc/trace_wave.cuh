// trace_wave.cuh — the wavefront tracing kernel (stage queues over a pool of
// paths) and its launch shapes, included by one translation unit per tracking
// mode (trace_wave_*.cu) so that its instantiations compile in parallel.
// trace_wave.cu holds the launch sequence (prepare, trace, finalize).
//
// The work of a chain falls into four stages:
//
//   track     a ray's next steps through the medium (sample_real_collision and
//             delta_transmittance, sky_trace.wgsl:405-475)
//   vertex    a primary ray that collided or reached the ground: the vertex and
//             its next sun sample (sky_trace.wgsl:566-608, 718-749)
//   continue  a vertex whose sun sample is decided: its NEE term, the next
//             direction, Russian roulette (sky_trace.wgsl:691-701, 728-767)
//   start     a chain that ended: its radiance, and the next sample's camera ray
//
// A block keeps its paths in shared memory and one queue of path numbers per
// stage.  A warp takes up to 32 paths from one queue, runs that one stage on
// them, tracks the rays that come out of it, and puts each path into the queue
// of the stage that it needs next.  So the lanes of a warp run the same code
// whatever pixel, chain or vertex their paths are at; nothing waits at a block
// barrier.  A warp leaves the tracking loop when few of its rays are still
// under way: those go to the track queue and continue in a fuller warp.
//
// What bounds it: instruction issue.  HBM and the tensor cores have no part in
// it (16 B leave the chip per cell, and a path is a chain of branches).  The
// ray loop (trace_ray.cuh) keeps each lane's path in registers and runs all event
// code once per ray: 9.5 of 32 lanes active per instruction, 7.9 G warp
// instructions and 7.42 ms for 42 M chains (128x64, 81 bands, 64 spp).  Here
// 22.6 lanes are active, for 4.9 G instructions at 86 % of the issue slots and 4.65
// ms; what is left is the rays' different lengths (tracking is two fifths) and
// the queues (a fifth).  What took it there: tracking right after the stage,
// instead of queueing every ray for it, 6.2 to 5.4 ms; staying with a stage, 5.15
// (instruction fetch was the first stall: the stages are large, and a scheduler's
// warps are in different ones); one copy of the rays' set-up for all stages,
// 4.87; products for the start's quotients, 4.84; the tracking loop's crossings
// and parking limits, 4.65.
//
// Each chain consumes its random stream in the plain kernel's order
// (trace_path, sky_trace.wgsl:703-776), so both kernels trace the same paths.
// Radiances are added to the job's cell sums by FP64 reductions in L2, in no
// fixed order (the sums agree with the plain kernel's to FP64 rounding).
//
// A launch is three kernels: prepare (zero the sums of jobs that do not
// accumulate, reset the work counter), trace, and finalize (mean film, XYZ
// and its variance, linear sRGB of every pixel of every job).

#pragma once

#include <algorithm>

#include "launch_limits.h"
#include "stage_queues.cuh"
#include "trace_common.cuh"

namespace sky {
namespace wave {

// Batches of a warp that count as one iteration of SkyTuning.iteration_limit (32
// chains take about 3.7 batches and 3 rays).  The batches are counted in 32 bits: a
// limit above 2^30 iterations, the default among them, is 2^32 - 1 batches, which take
// as many chains as 2^31 iterations of the ray loop.
constexpr uint64_t kBatchesPerIteration = 4;

// Rays still under way when a warp leaves the tracking loop and puts them back:
// most of a warp's rays end within a few steps, a few take many times that.  The
// fewer steps a queue entry costs, the more are left: merged layers (2.3 steps a
// ray) 8 -> 14 of 32 takes 4.74 to 4.65 ms (128x64, 81 bands, 64 spp), 20 4.68;
// the other modes, layer by layer (some 30 steps), 12 -> 26 takes 6.06 to 4.85 ms
// (64x32, 41 bands, 64 spp), 28 the same.
constexpr uint32_t kPark = 14, kParkLayered = 26;
// Rays that still have a crossing to make when a warp turns to its tentative
// collisions.
constexpr uint32_t kCrossing = 3;


// Blocks per SM.  A kernel shape is the warps of a block (SkyTuning.variant).
constexpr int kBlocksPerSm = 2;

// How a ray ended (Path B.y): a real collision at t, the boundary, or no ray
// at all (the chain's radiance is final; the path has no chain yet).
enum : uint32_t { kHit = 1u, kMiss = 2u, kOver = 3u, kFresh = 4u };

enum : uint32_t { kFlagShadow = 1u << 8, kFlagGround = 1u << 9, kFlagTop = 1u << 10 };

// A path in shared memory: rows of 16 bytes.
//   A  the ray's geometry: b, p, |o|^2, t_max
//   B  the tracker's state: t, two words of its own (how the ray ended, once it
//      has), the position in the random stream
//   C  the stream's keys of pixel and sample; band, flags and the tracker's
//      layer; job and the vertex's sun samples so far
//   D  vertex (ray origin) and throughput
//   E  direction and radiance
//   F  depth, cell, the vertex's NEE sum, the cosine of its sun sample
//   G  (H) the medium at the vertex: Rayleigh, total and species' scattering
// The row count is odd, so that the 16-byte accesses of neighbouring paths
// fall into different banks.
enum : uint32_t { kA = 0u, kB = 1u, kC = 2u, kD = 3u, kE = 4u, kF = 5u, kG = 6u, kH = 7u };
template <int kAer>
__host__ __device__ constexpr uint32_t path_rows() {
    return kAer == 1 ? 7u : 9u;
}

__host__ __device__ inline size_t pool_offset(uint32_t knots, uint32_t bands) {
    return align16(staged_medium_bytes(knots, bands));
}
// Dynamic shared memory of a block: staged medium, paths, queues.
template <int kAer>
__host__ __device__ inline size_t wave_smem_bytes(uint32_t knots, uint32_t bands, uint32_t paths) {
    return pool_offset(knots, bands) + size_t(paths) * path_rows<kAer>() * 16u + sizeof(Queues) +
           size_t(kQueues) * queue_slots(paths) * sizeof(uint16_t);
}

__device__ __forceinline__ Rng path_rng(const float4& C, uint32_t dim) {
    Rng r;
    r.k0 = as_u(C.x);
    r.k1 = as_u(C.y);
    r.k2 = (as_u(C.z) & 255u) * 1664525u + 1013904223u;
    r.dim = dim;
    return r;
}

// a / d and its remainder, from floor((2^32 - 1) / d).
__device__ __forceinline__ uint32_t quotient(uint32_t a, uint32_t d, uint32_t reciprocal, uint32_t& rest) {
    uint32_t q = __umulhi(a, reciprocal);
    rest = a - q * d;
    if (rest >= d) {
        ++q;
        rest -= d;
    }
    return q;
}

// Start of a ray's tracking: what of the tracker's state depends on the ray
// alone, and the first draws.  Fills B and the layer bits of C.z.
template <int kTracking>
__device__ __forceinline__ void track_begin(const DevScene& S, const RayGeo& g, float t_max, uint32_t band, Rng& rng,
                                            float4& B, uint32_t& meta, Counters& n) {
    if constexpr (kTracking == SKY_TRACKING_MERGED_LAYERS) {
        const MergedGrid G = merged_grid(S, band);
        int m = merged_layer_at(S, G, altitude_at(g, fminf(kRayEpsilonKm, t_max), S.ground_radius));
        int dir;
        const float t_seg = merged_crossing(G, g, m, 0.0f, t_max, dir);
        ++n.e[SKY_EVENT_SEGMENT];
        const float tau = -__logf(fmaxf(1.0f - rng.next(), 0.0000001f));
        B = make_float4(0.0f, tau, t_seg, as_f(rng.dim));
        meta |= (uint32_t(m) << 16) | (uint32_t(dir + 1) << 28);
    } else {
        B = make_float4(0.0f, -1.0f, as_f(0u), as_f(rng.dim));  // no optical depth drawn, no segment behind it
    }
}

// Track the warp's rays until at most `park` of them are under way.  Returns
// how the lane's ray ended (0: not yet), with t at its end.
template <int kTracking>
__device__ __forceinline__ uint32_t track_batch(const DevScene& S, const Medium& M, bool alive, const RayGeo& g,
                                                float t_max, uint32_t band, bool shadow, Rng& rng, float4& B,
                                                uint32_t& meta, Counters& n, bool& watchdog, uint32_t park) {
    const float2* sig_row = S.sigma_t + band * S.knot_count;
    const float4* cell_row = S.sig_cell + band * kFinderCells;
    float t = B.x;
    uint32_t ended = 0u;
    if constexpr (kTracking == SKY_TRACKING_MERGED_LAYERS) {
        // track_ray_merged: a step is the ray's crossings up to the segment that holds its
        // next tentative collision (or some of them), then that collision
        const MergedGrid G = merged_grid(S, band);
        int m = int((meta >> 16) & 0xfffu), dir = int(meta >> 28) - 1;
        float tau = B.y, t_seg = B.z;
        float maj = alive ? __ldg(G.maj + m) : 1.0f;
        for (uint32_t step = 0u; step < 4096u; ++step) {  // a ray crosses at most 2 x 1024 shells
            // the next tentative collision: one expression, which the compiler contracts into
            // the multiply-add that the plain kernel rounds with
            float next_t = 0.0f;
            if (alive) next_t = t + tau / maj;
            for (;;) {  // the crossings, until few rays have more to make (one each: +1.5 %)
                if (alive && !(next_t < t_seg)) {
                    if (dir == 0) {
                        ended = kMiss;
                        alive = false;
                    } else {
                        tau = fmaxf(tau - (t_seg - t) * maj, 0.0f);
                        t = t_seg;
                        m += dir;
                        t_seg = merged_crossing(G, g, m, t, t_max, dir);
                        maj = __ldg(G.maj + m);
                        ++n.e[SKY_EVENT_SEGMENT];
                        next_t = t + tau / maj;
                    }
                }
                if (__popc(__ballot_sync(kFull, alive && !(next_t < t_seg))) <= kCrossing) break;
            }
            if (alive && next_t < t_seg) {
                t = next_t;
                ++n.e[SKY_EVENT_TRACK_STEP];
                const float accept = rng.next() * maj;
                const float sig =
                    sigma_t_at(S, M.knot_z, M.finder, sig_row, cell_row, altitude_at(g, t, S.ground_radius));
                if (accept < sig) {
                    ended = kHit;
                    alive = false;
                } else {
                    tau = -__logf(fmaxf(1.0f - rng.next(), 0.0000001f));
                }
            }
            if (uint32_t(__popc(__ballot_sync(kFull, alive))) <= park) break;
        }
        B.x = t;
        B.y = tau;
        B.z = t_seg;
        meta = (meta & 0xffffu) | (uint32_t(m) << 16) | (uint32_t(dir + 1) << 28);
    } else {
        // track_ray's other modes: a step opens a segment if the ray is at one's
        // start, and makes one draw in it; rays park at a segment's start only
        const float* maj_row = S.majorants + band * S.layer_count;
        float tau = B.y, seg_end = 0.0f, maj = 1.0f;
        uint32_t guard = as_u(B.z);
        bool open = false;
        for (;;) {
            // segment restart: the step's draw, made before its segment is known so that the
            // two chains of arithmetic overlap; it counts (dim) only where it is used
            Rng ahead = rng;
            float lg = 0.0f;
            if constexpr (kTracking == SKY_TRACKING_SEGMENT_RESTART)
                lg = __logf(fmaxf(1.0f - ahead.next(), 0.0000001f));
            if (alive && !open) {
                if (t >= t_max) {
                    ended = kMiss;
                    alive = false;
                } else if (guard > 100000u) {
                    watchdog = true;
                    ended = shadow ? kHit : kMiss;
                    alive = false;
                } else {
                    ++guard;
                    uint32_t layer;
                    seg_end = next_segment_end(S, g, t, t_max, layer);
                    ++n.e[SKY_EVENT_SEGMENT];
                    maj = fmaxf(__ldg(maj_row + layer), 0.00000001f);
                    open = true;
                }
            }
            if (alive) {
                bool inside;
                if constexpr (kTracking == SKY_TRACKING_RESIDUAL_CARRY) {
                    if (tau < 0.0f) tau = -__logf(fmaxf(1.0f - rng.next(), 0.0000001f));
                    const float dt = tau / maj;
                    inside = !(t + dt >= seg_end);
                    if (inside) {
                        t = t + dt;
                        tau = -1.0f;
                    } else {
                        tau = fmaxf(tau - (seg_end - t) * maj, 0.0f);
                    }
                } else {
                    inside = !(t >= seg_end);
                    if (inside) {
                        rng.dim = ahead.dim;
                        t = t - lg / maj;
                        inside = !(t >= seg_end);
                    }
                }
                if (inside) {
                    ++n.e[SKY_EVENT_TRACK_STEP];
                    const float accept = rng.next() * maj;
                    const float sig =
                        sigma_t_at(S, M.knot_z, M.finder, sig_row, cell_row, altitude_at(g, t, S.ground_radius));
                    if (accept < sig) {
                        ended = kHit;
                        alive = false;
                    }
                } else {
                    t = seg_end;
                    open = false;
                }
            }
            const uint32_t active = __ballot_sync(kFull, alive);
            if (uint32_t(__popc(active)) <= park && __ballot_sync(kFull, alive && open) == 0u) break;
        }
        B.x = t;
        B.y = tau;
        B.z = as_f(guard);
    }
    if (ended) B.y = as_f(ended);
    B.w = as_f(rng.dim);
    return ended;
}

// kCount: count events (SkyDeviceOutputs.counters given).  Without it the
// counters are never read, so their increments compile away.
// kAer: aerosol species evaluated by the medium functions (1 or kSpecies,
// coefficients_at()).
template <int kTracking, int kPhase, int kWarps, bool kSingle, bool kCount, int kAer>
__global__ void __launch_bounds__(kWarps * 32, kBlocksPerSm)
    wave_kernel(const __grid_constant__ DevScene S, const __grid_constant__ DevLaunch L0,
                const DevJob* __restrict__ jobs, uint32_t num_jobs, unsigned long long total_chains, uint32_t paths,
                uint32_t used_paths, unsigned long long* __restrict__ work_counter,
                unsigned long long* __restrict__ counters, uint32_t* __restrict__ status, uint32_t batch_limit) {
    constexpr uint32_t kRows = path_rows<kAer>();
    extern __shared__ __align__(16) unsigned char smem[];
    float4* const pool = reinterpret_cast<float4*>(smem + pool_offset(S.knot_count, S.band_count));
    Queues* const Q = reinterpret_cast<Queues*>(pool + size_t(paths) * kRows);
    const StageQueues queues(Q, paths, used_paths);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = threadIdx.x; i < used_paths; i += blockDim.x)
        pool[i * kRows + kB] = make_float4(0.0f, as_f(kFresh), 0.0f, 0.0f);
    const Medium M = stage_medium(S, smem);  // ends with the block's only barrier
    Counters n;
    n.clear();
    bool watchdog = false;
    uint32_t idle = 0u, turn = (threadIdx.x >> 5) & 3u;
    uint32_t job_hint = 0u;  // the job of the last chains that the warp took: chains are taken in order

    for (uint32_t batch = 0u;;) {
        uint32_t stage, take, id;
        const Taken taken = queues.take(lane, turn, idle, batch, batch_limit, status, stage, take, id);
        if (taken == kOutOfWork) break;
        if (taken == kNothing) continue;
        const bool on = lane < take;
        float4* const P = pool + id * kRows;
        uint32_t next = kQNone;
        // the lane's ray: set up from its stage's origin and direction, or taken up where it was left
        bool tracing = false, set_up = false;
        V3 ray_org = mk(0.0f, 0.0f, 0.0f), ray_dir = ray_org;
        float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f), B = A;
        uint32_t meta = 0u;
        Rng rng;
        rng.k0 = rng.k1 = rng.k2 = rng.dim = 0u;

        if (stage == kQTrack) {
            if (on) {
                A = P[kA];
                B = P[kB];
                const float4 C = P[kC];
                meta = as_u(C.z);
                rng = path_rng(C, as_u(B.w));
                tracing = true;
            }
        } else if (stage == kQVertex) {
            if (on) {
                A = P[kA];
                B = P[kB];
                const float4 C = P[kC], D = P[kD], E = P[kE];
                meta = as_u(C.z);
                const uint32_t band = meta & 255u, job = as_u(C.w) & 0xffffu;
                uint32_t ls = as_u(C.w) >> 16;
                const DevLaunch& JL = job_launch<kSingle>(L0, jobs, job);
                V3 org = mk(D.x, D.y, D.z);
                const V3 dir = mk(E.x, E.y, E.z);
                bool ground = (meta & kFlagGround) != 0u, alive = true;
                if (!(meta & kFlagShadow)) {  // a new vertex
                    ls = 0u;
                    float thr = D.w;
                    ground = as_u(B.y) != kHit;
                    if (!ground) {
                        const RayGeo g{A.x, A.y, A.z};
                        org = madd(org, dir, B.x);
                        const float alt = altitude_at(g, B.x, S.ground_radius);
                        ++n.e[SKY_EVENT_SCATTER];
                        const Coeffs c = coefficients_at<kAer>(S, M, band, alt);
                        const bool medium = c.extinction > 0.0f && c.scattering > 0.0f;
                        if (medium) thr *= fminf(fmaxf(c.scattering / c.extinction, 0.0f), 1.0f);
                        if (!medium || thr <= 0.0f) {
                            alive = false;
                        } else {
                            P[kG] = make_float4(c.rayleigh, c.scattering, c.sca[0], c.sca[1]);
                            if (kAer > 1) P[kH] = make_float4(c.sca[2], c.sca[3], 0.0f, 0.0f);
                        }
                    } else {
                        ++n.e[SKY_EVENT_GROUND];
                        org = madd(org, dir, A.w);
                    }
                    P[kD] = make_float4(org.x, org.y, org.z, thr);
                    reinterpret_cast<float*>(&P[kF])[2] = 0.0f;  // the vertex's NEE sum
                }
                if (!alive) {
                    reinterpret_cast<float*>(&P[kE])[3] = fmaxf(E.w, 0.0f);
                    reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                    next = kQStart;
                } else {
                    // direct_sun_at_scatter (sky_trace.wgsl:566-585) and ground_radiance
                    // (:587-608), one shadow ray at a time
                    rng = path_rng(C, as_u(B.w));
                    const uint32_t lights = JL.direct_light_samples;
                    meta = band | kFlagShadow | (ground ? uint32_t(kFlagGround) : 0u);
                    next = kQContinue;
                    B = make_float4(0.0f, as_f(kHit), 0.0f, 0.0f);  // no sun: as a shadow ray that collides
                    while (ls < lights) {
                        ++ls;
                        const V3 ldir = sample_sun_cone(job_scene<kSingle>(S, jobs, job), rng);
                        ++n.e[SKY_EVENT_NEE];
                        float cos_sun = 0.0f;
                        if (ground) {
                            cos_sun = fmaxf(dot3(normalize_or_y(org), ldir), 0.0f);
                            if (!(cos_sun > 0.0f)) continue;
                        }
                        ray_org = madd(org, ldir, kRayEpsilonKm);
                        ray_dir = ldir;
                        reinterpret_cast<float*>(&P[kF])[3] = ground ? cos_sun : dot3(dir, ldir);
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
                const float4 C = P[kC], D = P[kD], E = P[kE], F = P[kF];
                B = P[kB];
                meta = as_u(C.z);
                const uint32_t band = meta & 255u, job = as_u(C.w) & 0xffffu, ls = as_u(C.w) >> 16;
                const DevLaunch& JL = job_launch<kSingle>(L0, jobs, job);
                const bool ground = (meta & kFlagGround) != 0u;
                V3 org = mk(D.x, D.y, D.z), dir = mk(E.x, E.y, E.z);
                float nee = F.z;
                Coeffs c;
                if (!ground) {
                    const float4 G = P[kG];
                    c.rayleigh = G.x;
                    c.scattering = G.y;
                    c.sca[0] = G.z;
                    c.sca[1] = c.sca[2] = c.sca[3] = 0.0f;
                    if (kAer > 1) {
                        const float4 H = P[kH];
                        c.sca[1] = G.w;
                        c.sca[2] = H.x;
                        c.sca[3] = H.y;
                    }
                    c.abs_total = 0.0f;
                    c.extinction = c.scattering;
                }
                if (as_u(B.y) == kMiss) {  // the sample's term, transmittance 1 (sky_trace.wgsl:566-608)
                    const float l_sun = M.bands[band].solar_radiance;
                    const float nee_mu = F.w;
                    nee += ground ? S.ground_albedo * kInvPi * l_sun * 1.0f * nee_mu / S.light_pdf
                                  : l_sun * 1.0f * mixed_phase<kAer>(S, c, band, nee_mu) / S.light_pdf;
                }
                const uint32_t lights = JL.direct_light_samples;
                if (ls < lights) {
                    reinterpret_cast<float*>(&P[kF])[2] = nee;
                    next = kQVertex;
                } else {
                    // the continuation (sky_trace.wgsl:728-767): each branch draws its
                    // angles, then one shared frame step turns them into the direction
                    // (orthonormal_basis + direction_from_frame, as direction_from_axis_mu
                    // and sample_cosine_hemisphere compute it), so that medium and ground
                    // lanes run that step together
                    rng = path_rng(C, as_u(B.w));
                    float thr = D.w, rad = E.w;
                    uint32_t depth = as_u(F.x);
                    rad += thr * (nee * (1.0f / float(lights)));
                    V3 nd = mk(0.0f, 1.0f, 0.0f), axis = dir;
                    float cos_t = 1.0f, sin_t = 0.0f, xi_phi = 0.0f, weight = 1.0f;
                    bool framed = true;
                    if (!ground) {
                        if (kPhase == SKY_PHASE_TABULATED) {
                            float mu;
                            weight = tabulated_mu<kAer>(S, c, band, rng, mu, xi_phi);
                            cos_t = fminf(fmaxf(mu, -1.0f), 1.0f);
                            sin_t = sqrtf(fmaxf(1.0f - cos_t * cos_t, 0.0f));
                        } else {
                            nd = sample_isotropic(rng);
                            weight = mixed_phase<kAer>(S, c, band, dot3(dir, nd)) / kIsotropicPdf;
                            framed = false;
                        }
                    } else {
                        axis = normalize_or_y(org);  // the ground normal
                        const float u = rng.next();
                        sin_t = sqrtf(u);
                        xi_phi = rng.next();
                        cos_t = sqrtf(fmaxf(1.0f - u, 0.0f));
                    }
                    V3 nrm = axis;
                    if (framed) {
                        V3 t, bt;
                        orthonormal_basis(axis, t, bt);
                        nrm = normalize_or_y(axis);
                        nd = direction_from_frame(nrm, t, bt, cos_t, sin_t, xi_phi);
                    }
                    bool alive = true;
                    if (ground) {
                        const float pdf = fmaxf(dot3(nrm, nd), 0.0f) * kInvPi;
                        const float cos_out = fmaxf(dot3(axis, nd), 0.0f);
                        if (pdf <= 0.0f || cos_out <= 0.0f) alive = false;
                        else thr *= S.ground_albedo * kInvPi * cos_out / pdf;
                    } else {
                        thr *= weight;
                    }
                    if (alive && depth >= JL.rr_start_depth) {  // russian_roulette (:691-701)
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
                        } else {
                            ++depth;
                        }
                    }
                    if (alive && depth >= JL.watchdog_limit) {
                        watchdog = true;
                        alive = false;
                    }
                    // what the next ray finds at its boundary may still end the chain, with this radiance
                    P[kD] = make_float4(org.x, org.y, org.z, thr);
                    P[kE] = make_float4(dir.x, dir.y, dir.z, rad);
                    reinterpret_cast<float*>(&P[kF])[0] = as_f(depth);
                    set_up = alive;
                    ray_org = org;
                    ray_dir = dir;
                    meta = band;
                    if (!alive) {
                        reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                        next = kQStart;
                    }
                }
            }
        } else {
            // the chains that ended
            float rad = 0.0f;
            uint32_t old_cell = 0u, old_job = 0u;
            const uint32_t state = on ? as_u(P[kB].y) : uint32_t(kFresh);
            if (state != kFresh) {
                const float4 C = P[kC], E = P[kE], F = P[kF];
                rad = E.w;
                old_cell = as_u(F.y);
                old_job = as_u(C.w) & 0xffffu;
                if (state == kMiss) {  // left through the top of the atmosphere
                    if (as_u(F.x) == 0u && dot3(mk(E.x, E.y, E.z), load3(job_scene<kSingle>(S, jobs, old_job).sun)) >=
                                               S.cos_max)
                        rad += P[kD].w * M.bands[as_u(C.z) & 255u].solar_radiance;
                    rad = fmaxf(rad, 0.0f);
                }
            }
            // the next samples of the launch, band-major (all pixels of a band, then the
            // next band), so that the warps of the chip work on one or two bands at a
            // time and that band's extinction row, merged grid and phase rows stay in L1;
            // the sums keep their pixel-major, band-minor layout
            unsigned long long base = 0u;
            if (lane == 0u) base = atomicAdd(work_counter, (unsigned long long)take);
            base = __shfl_sync(kFull, base, 0);
            const unsigned long long at = base + lane;
            const bool more = on && at < total_chains;
            uint32_t job = job_hint;
            if (!kSingle && more) {
                // the last job whose first chain is <= at: mostly that of the warp's last chains
                // (searching all jobs each time: 16 images of 128x64, 40 bands, 130.5
                // against 126.9 ms)
                uint32_t hi = num_jobs;
                if (job + 1u < hi && __ldg(&jobs[job + 1u].chain_begin) > at) hi = job + 1u;
                while (hi - job > 1u) {
                    const uint32_t mid = (job + hi) >> 1;
                    if (__ldg(&jobs[mid].chain_begin) <= at) job = mid;
                    else hi = mid;
                }
            }
            if (!kSingle) job_hint = __shfl_sync(kFull, job, 0);
            if (more) {
                const DevLaunch& JL = job_launch<kSingle>(L0, jobs, job);
                const unsigned long long rel = kSingle ? at : at - __ldg(&jobs[job].chain_begin);
                // cell and sample, band and pixel of the slab, row and column: quotients by products
                // with floor((2^k - 1) / divisor), which are at most one short
                uint32_t c = uint32_t(__umul64hi(rel, JL.spp_reciprocal));
                uint32_t sample = uint32_t(rel - (unsigned long long)c * JL.spp);
                if (sample >= JL.spp) {
                    ++c;
                    sample -= JL.spp;
                }
                uint32_t slab_pixel, px;
                const uint32_t band = quotient(c, JL.width * JL.rows, JL.pixels_reciprocal, slab_pixel);
                const uint32_t py = quotient(slab_pixel, JL.width, JL.width_reciprocal, px) + JL.row_begin;
                // the image pixel drives the random stream, the slab pixel indexes the sums
                rng.init(py * JL.width + px, JL.sample_offset + sample, band, JL.seed_lo, JL.seed_hi);
                const V3 dir = camera_dir(JL, px, py, rng);
                const V3 org = mk(0.0f, S.ground_radius + fmaxf(JL.observer_altitude, 0.0f), 0.0f);
                ++n.e[SKY_EVENT_CHAIN];
                meta = band;
                set_up = true;
                ray_org = org;
                ray_dir = dir;
                P[kC] = make_float4(as_f(rng.k0), as_f(rng.k1), as_f(band), as_f(job));
                P[kD] = make_float4(org.x, org.y, org.z, 1.0f);
                P[kE] = make_float4(dir.x, dir.y, dir.z, 0.0f);
                P[kF] = make_float4(as_f(0u), as_f(slab_pixel * S.band_count + band), 0.0f, 0.0f);
            }
            const uint32_t gone = __popc(__ballot_sync(kFull, on && !more));
            if (gone && lane == 0u) atomicSub(&Q->live, gone);
            if (rad != 0.0f) {  // the sums start at zero
                const DevJob& J = jobs[old_job];
                const double rd = double(rad);
                atomicAdd(J.cell_sum + old_cell, rd);
                double* sq = J.cell_sumsq;
                if (sq) atomicAdd(sq + old_cell, rd * rd);
            }
        }

        // the stages' rays: a shadow ray goes to the sun or leaves its vertex without one
        // (sky_trace.wgsl:574-577), an outgoing ray ends the chain where it meets no boundary
        // (:709-717).  One copy of this code for all stages: it is a third of theirs, and the
        // instruction caches are short of room.
        if (set_up) {
            const RayGeo g = ray_geo(ray_org, ray_dir);
            const bool shadow = (meta & kFlagShadow) != 0u;
            const uint32_t word = as_u(reinterpret_cast<const float*>(&P[kC])[3]);
            const DevLaunch& JL = job_launch<kSingle>(L0, jobs, word & 0xffffu);
            ++n.e[SKY_EVENT_BOUNDARY];
            float t_max;
            uint32_t boundary;
            bool ok = next_boundary(S, g, t_max, boundary);
            if (shadow) {
                ok = ok && boundary == 1u;
                if (!ok && (word >> 16) < JL.direct_light_samples) next = kQVertex;  // the next sample
            } else {
                const uint32_t max_orders = JL.max_orders;
                if (max_orders != 0u && as_u(reinterpret_cast<const float*>(&P[kF])[0]) >= max_orders) ok = false;
                if (boundary == 1u) meta |= kFlagTop;
                if (!ok) {
                    float* rad = reinterpret_cast<float*>(&P[kE]) + 3;
                    *rad = fmaxf(*rad, 0.0f);
                    reinterpret_cast<float*>(&P[kB])[1] = as_f(kOver);
                    next = kQStart;
                }
            }
            if (ok) {
                track_begin<kTracking>(S, g, t_max, meta & 255u, rng, B, meta, n);
                A = make_float4(g.b, g.p, g.r0sq, t_max);
                tracing = true;
            }
        }
        // track the rays at once, whatever stage they come from
        const uint32_t rays = __popc(__ballot_sync(kFull, tracing));
        if (rays) {
            const RayGeo g{A.x, A.y, A.z};
            // fewer of a small batch
            const uint32_t park = kTracking == SKY_TRACKING_MERGED_LAYERS ? min(kPark, rays / 2u)
                                                                          : min(kParkLayered, rays * 7u / 8u);
            const uint32_t ended = track_batch<kTracking>(S, M, tracing, g, A.w, meta & 255u,
                                                          (meta & kFlagShadow) != 0u, rng, B, meta, n, watchdog, park);
            if (tracing) {
                if (!ended) next = kQTrack;
                else if (meta & kFlagShadow) next = kQContinue;
                else next = ended == kMiss && (meta & kFlagTop) ? kQStart : kQVertex;
                if (next == kQTrack || next == kQVertex) P[kA] = A;
                P[kB] = B;
                reinterpret_cast<float*>(&P[kC])[2] = as_f(meta);
            }
        }

        queues.put(lane, next, id, status);
    }
    if (kCount) {
#pragma unroll
        for (int e = 0; e < SKY_EVENT_COUNT; ++e) {
            uint32_t v = n.e[e];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
            if (lane == 0u && v) atomicAdd(counters + e, (unsigned long long)v);
        }
    }
    if (__any_sync(kFull, watchdog) && lane == 0u) atomicOr(status, 1u);
}

// What a device offers a launch.
struct SharedRoom {
    int per_sm = 0, per_block = 0, reserved = 0;
    cudaError_t read() {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
        return e;
    }
    template <int kAer>
    bool fits(const WaveLaunch& w, uint32_t paths, int blocks) const {
        const size_t b = wave_smem_bytes<kAer>(w.scene.knot_count, w.scene.band_count, paths);
        return b <= size_t(per_block) && size_t(blocks) * (b + size_t(reserved)) <= size_t(per_sm);
    }
};

template <int kTracking, int kPhase, int kWarps, bool kSingle, bool kCount, int kAer>
cudaError_t launch_wave_shape(const WaveLaunch& w, cudaStream_t stream) {
    const void* k =
        reinterpret_cast<const void*>(wave_kernel<kTracking, kPhase, kWarps, kSingle, kCount, kAer>);
    constexpr uint32_t kThreads = kWarps * 32u;
    int per_sm = 0;
    SharedRoom room;
    cudaError_t e = room.read();
    if (e != cudaSuccess) return e;
    // paths of a block: a quarter more than its lanes (what waits in the queues while every
    // warp has a batch; a half more measured the same), fewer where the scene's tables leave
    // no room for that in two blocks per SM, in steps of 32
    uint32_t paths = kThreads * 5u / 4u;
    auto fits = [&](uint32_t p, int blocks) { return room.fits<kAer>(w, p, blocks); };
    while (paths > kThreads && !fits(paths, kBlocksPerSm)) paths -= 32u;
    if (!fits(paths, kBlocksPerSm)) {
        paths = kThreads * 5u / 4u;
        while (paths > 32u && !fits(paths, 1)) paths -= 32u;
    }
    const size_t smem = wave_smem_bytes<kAer>(w.scene.knot_count, w.scene.band_count, paths);
    if ((e = allow_shared_memory(k, smem)) != cudaSuccess) return e;
    // Prefer the smallest shared-memory carveout that holds two blocks: the rest of the
    // SM's L1/shared array caches the phase tables, extinction rows and merged grid.  A
    // hint: if the driver refuses it, the launch goes ahead with its own choice.
    const size_t need = size_t(fits(paths, kBlocksPerSm) ? kBlocksPerSm : 1) * (smem + size_t(room.reserved));
    const int pct = int(std::min<size_t>(100u, (need * 100u + size_t(room.per_sm) - 1u) / size_t(room.per_sm)));
    if (cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, std::max(pct, 1)) != cudaSuccess)
        (void)cudaGetLastError();  // clear the refused hint so the launch check does not see it
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem)) != cudaSuccess) return e;
    per_sm = std::max(per_sm, 1);
    if (w.max_blocks_per_sm) per_sm = std::min(per_sm, int(w.max_blocks_per_sm));
    // a warp of chains per block at least; a small render spreads its chains over the blocks
    const uint64_t want = (w.total_chains + 31u) / 32u;
    const uint32_t blocks = uint32_t(std::max<uint64_t>(1u, std::min<uint64_t>(uint64_t(per_sm) * uint64_t(w.sms), want)));
    const uint64_t share = ((w.total_chains + blocks - 1u) / blocks + 31u) / 32u * 32u;
    const uint32_t used = uint32_t(std::min<uint64_t>(paths, share));
    const uint32_t limit = uint32_t(std::min<uint64_t>(
        0xffffffffu, uint64_t(w.iteration_limit ? w.iteration_limit : kMaxIterations) * kBatchesPerIteration));
    wave_kernel<kTracking, kPhase, kWarps, kSingle, kCount, kAer><<<blocks, kThreads, smem, stream>>>(
        w.scene, w.launch0, w.jobs, w.num_jobs, w.total_chains, paths, used, w.work_counter, w.counters, w.status,
        limit);
    return cudaGetLastError();
}

template <int kTracking, int kPhase, bool kSingle, bool kCount, int kAer>
cudaError_t launch_wave_variant(const WaveLaunch& w, cudaStream_t stream) {
    // Where the tables leave room for one block of a shape only, the shape of most warps runs
    // for it (256 bands, 1000 layers, four species, 16.8 M chains: one block of 12 warps 3.65,
    // of 16 3.01 ms; one species 3.54, 2.89).
    uint32_t variant = w.variant;
    if (variant < 2u) {
        SharedRoom room;
        const cudaError_t e = room.read();
        if (e != cudaSuccess) return e;
        if (!room.fits<kAer>(w, variant == 0u ? 12u * 32u : 8u * 32u, kBlocksPerSm)) variant = 2u;
    }
    switch (variant) {
        case 0: return launch_wave_shape<kTracking, kPhase, 12, kSingle, kCount, kAer>(w, stream);
        case 1: return launch_wave_shape<kTracking, kPhase, 8, kSingle, kCount, kAer>(w, stream);
        case 2: return launch_wave_shape<kTracking, kPhase, 16, kSingle, kCount, kAer>(w, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <int kTracking, int kPhase, int kAer>
cudaError_t launch_wave_species(const WaveLaunch& w, cudaStream_t stream) {
    if (w.num_jobs == 1u)
        return w.counters ? launch_wave_variant<kTracking, kPhase, true, true, kAer>(w, stream)
                          : launch_wave_variant<kTracking, kPhase, true, false, kAer>(w, stream);
    return w.counters ? launch_wave_variant<kTracking, kPhase, false, true, kAer>(w, stream)
                      : launch_wave_variant<kTracking, kPhase, false, false, kAer>(w, stream);
}

template <int kTracking, int kPhase>
cudaError_t launch_wave_mode(const WaveLaunch& w, cudaStream_t stream) {
    if (w.aerosol_species == 1u) return launch_wave_species<kTracking, kPhase, 1>(w, stream);
    if (w.aerosol_species == kSpecies) return launch_wave_species<kTracking, kPhase, int(kSpecies)>(w, stream);
    return cudaErrorInvalidValue;
}

// The kernels of one tracking mode, both phase samplings.
template <int kTracking>
cudaError_t launch_wave_tracking(const WaveLaunch& w, cudaStream_t stream) {
    if (w.phase_sampling == SKY_PHASE_TABULATED) return launch_wave_mode<kTracking, SKY_PHASE_TABULATED>(w, stream);
    if (w.phase_sampling == SKY_PHASE_ISOTROPIC) return launch_wave_mode<kTracking, SKY_PHASE_ISOTROPIC>(w, stream);
    return cudaErrorInvalidValue;
}

}  // namespace wave
}  // namespace sky
