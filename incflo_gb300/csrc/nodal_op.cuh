// The nodal operator at one node, for the kernels that evaluate it cell by cell.
#pragma once

#include "gbp_internal.cuh"

namespace gbp {

// ---------------------------------------------------------------------------------------
// operator at one node
// ---------------------------------------------------------------------------------------
template <typename T>
struct NodalOp;

// FP64: the isotropic form sums sigma-weighted far-corner sums and subtracts the centre once
// (fewest FP64 instructions; FP64 issue rate, not HBM, bounds these kernels on GB300).
template <>
struct NodalOp<double> {
    template <bool ISO, typename I>
    __device__ __forceinline__ static double apply(const double* __restrict__ x, const double* __restrict__ s,
                                                   I c, I sy, I sz,
                                                   const NodalGeom& g, double& diag)
    {
        const double xc = x[c];
        double acc = 0.0, ssum = 0.0;
#pragma unroll
        for (int cz = 0; cz < 2; ++cz)
#pragma unroll
            for (int cy = 0; cy < 2; ++cy)
#pragma unroll
                for (int cx = 0; cx < 2; ++cx) {
                    const I cell = c + (cx - 1) + (cy - 1) * sy + (cz - 1) * sz;
                    const double sg = s[cell];
                    const I ox = cx ? 1 : -1, oy = cy ? sy : -sy, oz = cz ? sz : -sz;
                    ssum += sg;
                    if (ISO) {
                        double S = (x[c + ox + oy] + x[c + ox + oz]) +
                                   (x[c + oy + oz] + x[c + ox + oy + oz]);
                        acc = fma(sg, S, acc);
                    } else {
                        double t = g.K[1] * (x[c + ox] - xc) + g.K[2] * (x[c + oy] - xc) +
                                   g.K[4] * (x[c + oz] - xc) + g.K[3] * (x[c + ox + oy] - xc) +
                                   g.K[5] * (x[c + ox + oz] - xc) + g.K[6] * (x[c + oy + oz] - xc) +
                                   g.K[7] * (x[c + ox + oy + oz] - xc);
                        acc = fma(sg, t, acc);
                    }
                }
        diag = g.K[0] * ssum;
        if (ISO) return g.K[3] * fma(-4.0 * xc, ssum, acc);
        return acc;
    }
};

// FP32: explicit differences to the centre keep the rounding error proportional to the
// local variation of x rather than to x itself.
template <>
struct NodalOp<float> {
    template <bool ISO, typename I>
    __device__ __forceinline__ static float apply(const float* __restrict__ x, const float* __restrict__ s,
                                                  I c, I sy, I sz,
                                                  const NodalGeom& g, float& diag)
    {
        const float xc = x[c];
        float acc = 0.f, ssum = 0.f;
        const float k1 = (float)g.K[1], k2 = (float)g.K[2], k4 = (float)g.K[4], k3 = (float)g.K[3],
                    k5 = (float)g.K[5], k6 = (float)g.K[6], k7 = (float)g.K[7];
#pragma unroll
        for (int cz = 0; cz < 2; ++cz)
#pragma unroll
            for (int cy = 0; cy < 2; ++cy)
#pragma unroll
                for (int cx = 0; cx < 2; ++cx) {
                    const I cell = c + (cx - 1) + (cy - 1) * sy + (cz - 1) * sz;
                    const float sg = s[cell];
                    const I ox = cx ? 1 : -1, oy = cy ? sy : -sy, oz = cz ? sz : -sz;
                    ssum += sg;
                    if (ISO) {
                        float S = ((x[c + ox + oy] - xc) + (x[c + ox + oz] - xc)) +
                                  ((x[c + oy + oz] - xc) + (x[c + ox + oy + oz] - xc));
                        acc = fmaf(sg, S, acc);
                    } else {
                        float t = k1 * (x[c + ox] - xc) + k2 * (x[c + oy] - xc) +
                                  k4 * (x[c + oz] - xc) + k3 * (x[c + ox + oy] - xc) +
                                  k5 * (x[c + ox + oz] - xc) + k6 * (x[c + oy + oz] - xc) +
                                  k7 * (x[c + ox + oy + oz] - xc);
                        acc = fmaf(sg, t, acc);
                    }
                }
        diag = (float)g.K[0] * ssum;
        if (ISO) return (float)g.K[3] * acc;
        return acc;
    }
};

// Smoother weight / diagonal. A Jacobi smoother only needs an approximate reciprocal, so the
// FP64 path uses the single-precision reciprocal when the diagonal is in range.
__device__ __forceinline__ double approx_recip(double d)
{
    double a = fabs(d);
    if (a > 1e-30 && a < 1e30) return (double)__frcp_rn((float)d);
    return 1.0 / d;
}
__device__ __forceinline__ float approx_recip(float d) { return __frcp_rn(d); }

}  // namespace gbp
