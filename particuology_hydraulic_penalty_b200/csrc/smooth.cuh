// The smooth solid fraction of the adjoint: every sub-sample of a cell at distance d from a sphere's
// centre contributes sigma((r - d) / eps), sigma the logistic function, instead of the reference's
// inside test (psc3d.py:79-90).
#pragma once

#include "collide.cuh"

namespace psc {

// Beyond |z| = 40 the logistic function is 0 or 1 to the last bit of a double sum of samples
// (e^-40 < 2^-57), and its derivative counts for nothing.
constexpr double kSmoothFlat = 40.0;

// e^-|z| of sample distance d: sigma(z) = 1/(1+t) for z >= 0, t/(1+t) else; sigma' = t/(1+t)^2.
struct SmoothSample {
    double t, inv;  // inv = 1 / (1 + t)
};
__device__ __forceinline__ SmoothSample smooth_sample(double z) {
    SmoothSample s;
    s.t = exp(-fabs(z));
    s.inv = __drcp_rn(1.0 + s.t);
    return s;
}

// Where every sample of the cell is flat: +1 (all inside), -1 (all outside), else 0.  The samples lie
// within sqrt(3) (1/2 - 1/(2S)) of the cell's centre.
__device__ __forceinline__ int smooth_side(int32_t ix, int32_t iy, int32_t iz, double px, double py, double pz,
                                           double r, int S, double inv_eps) {
    const double dx = (double)ix + 0.5 - px, dy = (double)iy + 0.5 - py, dz = (double)iz + 0.5 - pz;
    const double d = sqrt(dx * dx + dy * dy + dz * dz);
    const double h = 0.8661 * (1.0 - 1.0 / (double)S) + 1.0e-9;
    if ((r - d - h) * inv_eps > kSmoothFlat) return 1;
    if ((r - d + h) * inv_eps < -kSmoothFlat) return -1;
    return 0;
}

// Mean of sigma over the S^3 samples (NS = S as a compile-time constant, or 0).
template <int NS>
__device__ __forceinline__ double smooth_alpha(int32_t ix, int32_t iy, int32_t iz, double px, double py, double pz,
                                               double r, int subsamples, double inv_eps) {
    const int S = NS > 0 ? NS : subsamples;
    const int side = smooth_side(ix, iy, iz, px, py, pz, r, S, inv_eps);
    if (side != 0) return side > 0 ? 1.0 : 0.0;
    const double Sd = (double)S, invS = 1.0 / Sd;
    double acc = 0.0;
    for (int a = 0; a < S; ++a) {
        const double dx = ((double)ix + ((double)a + 0.5) * invS) - px;
        for (int b = 0; b < S; ++b) {
            const double dy = ((double)iy + ((double)b + 0.5) * invS) - py;
            const double dxy = dx * dx + dy * dy;
#pragma unroll
            for (int c = 0; c < (NS > 0 ? NS : S); ++c) {
                const double dz = ((double)iz + ((double)c + 0.5) * invS) - pz;
                const double z = (r - sqrt(dxy + dz * dz)) * inv_eps;
                const SmoothSample s = smooth_sample(z);
                acc += z >= 0.0 ? s.inv : s.t * s.inv;
            }
        }
    }
    return acc / (Sd * Sd * Sd);
}

// Sums over the samples of sigma' / eps (gr) and of sigma' / eps times the unit vector from the centre
// (gx, gy, gz): the derivatives of S^3 alpha by r and by the centre.
template <int NS>
__device__ __forceinline__ void smooth_gradient(int32_t ix, int32_t iy, int32_t iz, double px, double py, double pz,
                                                double r, int subsamples, double inv_eps, double& gx, double& gy,
                                                double& gz, double& gr) {
    const int S = NS > 0 ? NS : subsamples;
    gx = gy = gz = gr = 0.0;
    if (smooth_side(ix, iy, iz, px, py, pz, r, S, inv_eps) != 0) return;
    const double invS = 1.0 / (double)S;
    for (int a = 0; a < S; ++a) {
        const double dx = ((double)ix + ((double)a + 0.5) * invS) - px;
        for (int b = 0; b < S; ++b) {
            const double dy = ((double)iy + ((double)b + 0.5) * invS) - py;
            const double dxy = dx * dx + dy * dy;
#pragma unroll
            for (int c = 0; c < (NS > 0 ? NS : S); ++c) {
                const double dz = ((double)iz + ((double)c + 0.5) * invS) - pz;
                const double d2 = dxy + dz * dz;
                const double dinv = d2 > 1.0e-24 ? rsqrt(d2) : 0.0;
                const SmoothSample s = smooth_sample((r - d2 * dinv) * inv_eps);
                const double ds = s.t * s.inv * s.inv * inv_eps;
                gr += ds;
                gx += ds * dx * dinv;
                gy += ds * dy * dinv;
                gz += ds * dz * dinv;
            }
        }
    }
}

// Launches KERNEL<S> for the subsample counts 1 .. 6, KERNEL<0> for others.
#define PSC_BY_SUBSAMPLES(S, KERNEL, ...)      \
    switch (S) {                               \
        case 1: KERNEL<1> __VA_ARGS__; break;  \
        case 2: KERNEL<2> __VA_ARGS__; break;  \
        case 3: KERNEL<3> __VA_ARGS__; break;  \
        case 4: KERNEL<4> __VA_ARGS__; break;  \
        case 5: KERNEL<5> __VA_ARGS__; break;  \
        case 6: KERNEL<6> __VA_ARGS__; break;  \
        default: KERNEL<0> __VA_ARGS__; break; \
    }

}  // namespace psc
