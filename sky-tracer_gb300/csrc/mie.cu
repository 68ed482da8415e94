// mie.cu — the Mie phase-table bake of scripts/bake_opac_data.py:103-121 and
// :192-204: for one aerosol species, the phase function on the cube-root mu
// grid averaged over a lognormal size distribution with scattering cross
// section weights,
//
//   p(mu) = sum_r w_r sigma_sca(r) p_r(mu) / sum_r w_r sigma_sca(r),
//
// where p_r is a sphere's unpolarised phase function normalised to 1 over the
// sphere.  The reference evaluates each sphere with miepython (efficiencies
// and i_unpolarized, norm="one"); miepython is not vendored and its version
// is not pinned, so the sphere is computed here from the published Mie series
// (Bohren & Huffman, "Absorption and Scattering of Light by Small Particles",
// 1983, appendix A, BHMIE; term count after Wiscombe, Appl. Opt. 19, 1505,
// 1980).  Since sigma_sca p_r = (|S1|^2 + |S2|^2) / (2 k^2), the average
// needs only the amplitude functions and Q_sca.
//
// Three kernels, over (band, radius) items taken from the largest radius down,
// so that the longest ones start first.
//
//   recurrences   what is sequential in n, one thread per item and chain: the
//                 logarithmic derivative D_n(mx) downward from max(N, |mx|) + 16,
//                 and the Riccati-Bessel functions psi_n, chi_n upward
//   coefficients  a_n, b_n of every n, a warp per item: stored in FP32
//                 pre-multiplied by (2n+1)/(n(n+1)), with Q_sca, Q_ext and the
//                 asymmetry parameter
//   angles        S1, S2 in FP32 (pi_n, tau_n recurrences), a block per band and
//                 share of its radii, four mu bins per thread whose FP64
//                 accumulators of w (|S1|^2 + |S2|^2) / (2 k^2) stay in registers
//
// What bounds them: FP64, at two operations per clock and SM, and in the first
// kernel the length of the longest item's chain (a warp's FP64 instruction takes
// 64 cycles of its scheduler's unit).  The series was one thread per item, some
// 250 FP64 instructions per term on that chain: 4.35 ms for 41 bands x 300 radii
// (waso).  With only the recurrences on it, the derivative's reciprocal by its
// squared modulus (one division instead of Smith's three), and the two chains in
// warps of their own: 0.41 ms and 0.34 ms for the coefficients.  The angles took 0.72
// ms when each item's block converted its bins to mu, squared four sums in FP64
// and added to L2 once per bin: 0.50 ms.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "launch_limits.h"
#include "mie_kernels.h"

namespace sky {
namespace {

struct Cd {
    double re, im;
};
__device__ __forceinline__ Cd cd(double re, double im) { return Cd{re, im}; }
__device__ __forceinline__ Cd operator+(Cd a, Cd b) { return cd(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ Cd operator-(Cd a, Cd b) { return cd(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ Cd operator*(Cd a, Cd b) { return cd(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
__device__ __forceinline__ Cd operator*(double s, Cd a) { return cd(s * a.re, s * a.im); }
// Smith's division, robust to the large magnitudes of xi_n beyond n ~ x.
__device__ __forceinline__ Cd operator/(Cd a, Cd b) {
    if (fabs(b.re) >= fabs(b.im)) {
        const double r = b.im / b.re, d = b.re + r * b.im;
        return cd((a.re + r * a.im) / d, (a.im - r * a.re) / d);
    }
    const double r = b.re / b.im, d = b.im + r * b.re;
    return cd((a.re * r + a.im) / d, (a.im * r - a.re) / d);
}
__device__ __forceinline__ double norm2(Cd a) { return a.re * a.re + a.im * a.im; }

// 1 / b.  By the squared modulus where that neither overflows nor underflows.
__device__ __forceinline__ Cd reciprocal(Cd b) {
    const double m = norm2(b);
    if (m > 1e-280 && m < 1e280) {
        const double r = 1.0 / m;
        return cd(b.re * r, -b.im * r);
    }
    return cd(1.0, 0.0) / b;
}

// Item of place i in the order of descending radii.
__device__ __forceinline__ uint32_t item_at(uint32_t i, uint32_t bands, uint32_t radii) {
    const uint32_t r = radii - 1u - i / bands;
    return (i % bands) * radii + r;
}

// Warp 0 of a block runs the derivative's recurrence of 32 items, warp 1 the
// Riccati-Bessel functions'.
__global__ void __launch_bounds__(64) mie_recurrences_kernel(const MieItem* __restrict__ items, uint32_t bands,
                                                             uint32_t radii, double2* __restrict__ series,
                                                             double2* __restrict__ riccati) {
    const uint32_t place = blockIdx.x * 32u + (threadIdx.x & 31u);
    if (place >= bands * radii) return;
    const uint32_t i = item_at(place, bands, radii);
    const MieItem it = items[i];
    const double x = it.x;
    if (threadIdx.x < 32u) {
        // D_{n-1} = n/(mx) - 1/(D_n + n/(mx)), D_nmx = 0
        const Cd inv_mx = cd(1.0, 0.0) / (x * cd(it.m_re, it.m_im));
        double2* D = series + it.off + i;
        Cd d = cd(0.0, 0.0);
        for (uint32_t n = it.dterms; n >= 1u; --n) {
            const Cd t = double(n) * inv_mx;
            d = t - reciprocal(d + t);
            if (n <= it.terms + 1u) D[n - 1u] = make_double2(d.re, d.im);
        }
    } else {
        double2* R = riccati + it.off + i;  // terms + 1 of an item: psi_n, chi_n from n = 0
        double psi0 = cos(x), psi1 = sin(x), chi0 = -sin(x), chi1 = cos(x);
        R[0] = make_double2(psi1, chi1);
        for (uint32_t n = 1u; n <= it.terms; ++n) {
            const double rn = double(n);
            const double psi = (2.0 * rn - 1.0) * psi1 / x - psi0;
            const double chi = (2.0 * rn - 1.0) * chi1 / x - chi0;
            R[n] = make_double2(psi, chi);
            psi0 = psi1;
            psi1 = psi;
            chi0 = chi1;
            chi1 = chi;
        }
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The coefficients of a term in the 16 bytes of its D_n.
__device__ __forceinline__ double2 pack(float a, float b, float c, float d) {
    return make_double2(__hiloint2double(__float_as_int(b), __float_as_int(a)),
                        __hiloint2double(__float_as_int(d), __float_as_int(c)));
}

// A warp per item, lane l the terms l + 1, l + 33, ...  A lane reads D_n and writes the
// term's coefficients over it (arrays of their own took half as much memory again).
__global__ void __launch_bounds__(128) mie_coefficients_kernel(const MieItem* __restrict__ items, uint32_t bands,
                                                               uint32_t radii, double2* __restrict__ series,
                                                               const double2* __restrict__ riccati,
                                                               double* __restrict__ q) {
    const uint32_t place = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (place >= bands * radii) return;  // whole warps
    const uint32_t i = item_at(place, bands, radii);
    const MieItem it = items[i];
    const double x = it.x;
    const Cd m = cd(it.m_re, it.m_im);
    const Cd inv_m = cd(1.0, 0.0) / m;
    double2* const D = series + it.off + i;
    const double2* R = riccati + it.off + i;
    double qsca = 0.0, qext = 0.0, gsum = 0.0;
    Cd a_end = cd(0.0, 0.0), b_end = cd(0.0, 0.0);  // of the 32 terms before
    for (uint32_t n0 = 0u; n0 < it.terms; n0 += 32u) {
        const uint32_t n = n0 + lane + 1u;
        Cd an = cd(0.0, 0.0), bn = cd(0.0, 0.0);
        const double rn = double(n);
        if (n <= it.terms) {
            const double2 r = R[n], r1 = R[n - 1u], dn2 = D[n];
            const double psi = r.x, psi1 = r1.x;
            const Cd xi = cd(psi, -r.y), xi1 = cd(psi1, -r1.y);
            const Cd dn = cd(dn2.x, dn2.y);
            const Cd ta = dn * inv_m + cd(rn / x, 0.0);
            const Cd tb = m * dn + cd(rn / x, 0.0);
            an = (psi * ta - cd(psi1, 0.0)) / (ta * xi - xi1);
            bn = (psi * tb - cd(psi1, 0.0)) / (tb * xi - xi1);
            const double fn = (2.0 * rn + 1.0) / (rn * (rn + 1.0));
            D[n] = pack(float(fn * an.re), float(fn * an.im), float(fn * bn.re), float(fn * bn.im));
            qsca += (2.0 * rn + 1.0) * (norm2(an) + norm2(bn));
            qext += (2.0 * rn + 1.0) * (an.re + bn.re);
            gsum += fn * (an.re * bn.re + an.im * bn.im);
        }
        // asymmetry: (n-1)(n+1)/n Re(a_{n-1} a_n* + b_{n-1} b_n*) + (2n+1)/(n(n+1)) Re(a_n b_n*)
        auto before = [&](double v, double end) {
            const double u = __shfl_up_sync(0xffffffffu, v, 1);
            return lane == 0u ? end : u;
        };
        const Cd a_prev = cd(before(an.re, a_end.re), before(an.im, a_end.im));
        const Cd b_prev = cd(before(bn.re, b_end.re), before(bn.im, b_end.im));
        if (n > 1u && n <= it.terms) {
            const double rm = rn - 1.0;
            gsum += rm * (rm + 2.0) / (rm + 1.0) *
                    (a_prev.re * an.re + a_prev.im * an.im + b_prev.re * bn.re + b_prev.im * bn.im);
        }
        a_end = cd(__shfl_sync(0xffffffffu, an.re, 31), __shfl_sync(0xffffffffu, an.im, 31));
        b_end = cd(__shfl_sync(0xffffffffu, bn.re, 31), __shfl_sync(0xffffffffu, bn.im, 31));
    }
    qsca = warp_sum(qsca);
    qext = warp_sum(qext);
    gsum = warp_sum(gsum);
    if (lane == 0u) {
        const double x2 = x * x;
        qsca *= 2.0 / x2;
        q[3 * i] = qsca;
        q[3 * i + 1] = qext * 2.0 / x2;
        q[3 * i + 2] = qsca > 0.0 ? gsum * 4.0 / (x2 * qsca) : 0.0;
    }
}

// v^2 added to a sum kept as an unevaluated pair of floats, exactly but for the
// rounding of the small part (the product by an FMA, the sum by Knuth's two-sum).
__device__ __forceinline__ void add_square(float& hi, float& lo, float v) {
    const float p = __fmul_rn(v, v), e = __fmaf_rn(v, v, -p);
    const float t = __fadd_rn(hi, p), b = __fsub_rn(t, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fadd_rn(__fsub_rn(hi, __fsub_rn(t, b)), __fsub_rn(p, b)), e));
    hi = t;
}

// Band blockIdx.x, radii blockIdx.y, + gridDim.y, ..., tiles of bins blockIdx.z, + gridDim.z, ...
constexpr uint32_t kAngleThreads = 256, kAngleBins = 4;
__global__ void __launch_bounds__(kAngleThreads) mie_angles_kernel(const MieItem* __restrict__ items, uint32_t radii,
                                                                   const float4* __restrict__ series, uint32_t bins,
                                                                   double* __restrict__ phase_acc) {
    extern __shared__ float4 coef[];
    constexpr uint32_t kTile = kAngleThreads * kAngleBins;
    for (uint32_t tile = blockIdx.z; uint64_t(tile) * kTile < bins; tile += gridDim.z) {
        float mu[kAngleBins];
        double acc[kAngleBins];
    #pragma unroll
        for (uint32_t k = 0; k < kAngleBins; ++k) {
            const uint32_t j = (tile * kAngleBins + k) * kAngleThreads + threadIdx.x;
            const double u = (double(j) + 0.5) / double(bins);
            mu[k] = float(1.0 - 2.0 * u * u * u);  // cube-root grid (bake_opac_data.py:99-101)
            acc[k] = 0.0;
        }
        for (uint32_t r = blockIdx.y; r < radii; r += gridDim.y) {
            const MieItem it = items[size_t(blockIdx.x) * radii + r];
            const uint32_t N = it.terms;
            __syncthreads();
            const float4* terms = series + it.off + size_t(blockIdx.x) * radii + r + 1u;  // of n = 1, 2, ...
            for (uint32_t n = threadIdx.x; n < N; n += blockDim.x) coef[n] = terms[n];
            __syncthreads();
            const double scale = it.weight / (2.0 * it.k * it.k);  // w / (2 k^2)
            float pi0[kAngleBins], pi1[kAngleBins], s1r[kAngleBins], s1i[kAngleBins], s2r[kAngleBins], s2i[kAngleBins];
    #pragma unroll
            for (uint32_t k = 0; k < kAngleBins; ++k) {
                pi0[k] = 0.0f;
                pi1[k] = 1.0f;
                s1r[k] = s1i[k] = s2r[k] = s2i[k] = 0.0f;
            }
            for (uint32_t n = 1u; n <= N; ++n) {
                const float rn = float(n);
                const float4 c = coef[n - 1u];
    #pragma unroll
                for (uint32_t k = 0; k < kAngleBins; ++k) {
                    const float pi = pi1[k];
                    const float tau = rn * mu[k] * pi - (rn + 1.0f) * pi0[k];
                    s1r[k] = fmaf(c.x, pi, fmaf(c.z, tau, s1r[k]));
                    s1i[k] = fmaf(c.y, pi, fmaf(c.w, tau, s1i[k]));
                    s2r[k] = fmaf(c.x, tau, fmaf(c.z, pi, s2r[k]));
                    s2i[k] = fmaf(c.y, tau, fmaf(c.w, pi, s2i[k]));
                    pi1[k] = ((2.0f * rn + 1.0f) * mu[k] * pi - (rn + 1.0f) * pi0[k]) / rn;
                    pi0[k] = pi;
                }
            }
    #pragma unroll
            for (uint32_t k = 0; k < kAngleBins; ++k) {
                float hi = 0.0f, lo = 0.0f;
                add_square(hi, lo, s1r[k]);
                add_square(hi, lo, s1i[k]);
                add_square(hi, lo, s2r[k]);
                add_square(hi, lo, s2i[k]);
                acc[k] += scale * (double(hi) + double(lo));
            }
        }
    #pragma unroll
        for (uint32_t k = 0; k < kAngleBins; ++k) {
            const uint32_t j = (tile * kAngleBins + k) * kAngleThreads + threadIdx.x;
            if (j < bins) atomicAdd(phase_acc + size_t(blockIdx.x) * bins + j, acc[k]);
        }
    }
}

}  // namespace

cudaError_t launch_mie_bake(const MieItem* items, uint32_t bands, uint32_t radii, uint32_t max_terms,
                            double2* series, double2* riccati, double* q, uint32_t bins, double* phase_acc,
                            uint32_t sms, cudaStream_t stream) {
    const uint32_t count = bands * radii;
    if (count == 0) return cudaSuccess;
    mie_recurrences_kernel<<<(count + 31u) / 32u, 64, 0, stream>>>(items, bands, radii, series, riccati);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    mie_coefficients_kernel<<<(count + 3u) / 4u, 128, 0, stream>>>(items, bands, radii, series, riccati, q);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const size_t smem = size_t(max_terms) * sizeof(float4);
    if ((e = allow_shared_memory(reinterpret_cast<const void*>(mie_angles_kernel), smem)) != cudaSuccess) return e;
    // four blocks per SM: the radii of a band in shares that each hold large and small ones
    const uint32_t tiles = uint32_t((uint64_t(bins) + kAngleThreads * kAngleBins - 1u) / (kAngleThreads * kAngleBins));
    const uint64_t each = uint64_t(bands) * tiles;
    const uint32_t shares = std::min(radii, std::max(1u, uint32_t((4u * sms + each - 1u) / each)));
    mie_angles_kernel<<<dim3(bands, shares, std::min(tiles, 65535u)), kAngleThreads, smem, stream>>>(
        items, radii, reinterpret_cast<const float4*>(series), bins, phase_acc);
    return cudaGetLastError();
}

}  // namespace sky
