// Device pieces of the Vegas integrator shared by the DIS terms (dis.cu) and the BK K2+Kf
// integral (k2kf_vegas.cu): the grid re-binning of _adapt_vegas_edges
// (numerics/integration.py:804-866) and the inverse-variance combination of the iteration
// estimates with the convergence test (:510-582).  Both run in one CTA per integral, in a
// fixed order, so results are bit-reproducible.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nlo {
namespace vegas {

// Slots after the edges [D][bins+1] of a per-integral state.
enum StateSlot {
    kStSumWeightedEst = 0,  // sum of estimate / variance over reported iterations
    kStSumWeights = 1,      // sum of 1 / variance
    kStValue = 2,
    kStError = 3,
    kStEvals = 4,
    kStIterations = 5,
    kStConverged = 6,
    kStLastEstimate = 7,
    kStLastVariance = 8,
    kStSlots = 16,
};

// New edges of every dimension from the |w| histogram and the bin counts: importance =
// hist / max(count, 1), three-point smoothing (two at the ends), + DBL_EPSILON, equal-mass
// re-binning of the cumulative importance against the old edges; the end edges stay 0 and 1.
// Called by all threads of the CTA; smooth [D*bins], cum [D*(bins+1)] and next [D*(bins+1)]
// are shared-memory scratch.  edges is read and then overwritten.
__device__ inline void rebin(double* edges, const double* hist, const int32_t* counts, int D, int bins,
                             double* smooth, double* cum, double* next)
{
    for (int k = threadIdx.x; k < D * bins; k += blockDim.x) {
        const int d = k / bins, b = k % bins;
        auto imp = [&](int q) {
            const int n = counts[d * bins + q];
            return hist[d * bins + q] / (double)(n > 1 ? n : 1);
        };
        double v;
        if (b == 0)
            v = (imp(0) + imp(1)) / 2.0;
        else if (b == bins - 1)
            v = (imp(bins - 2) + imp(bins - 1)) / 2.0;
        else
            v = (imp(b - 1) + imp(b) + imp(b + 1)) / 3.0;
        smooth[k] = v + 2.220446049250313e-16;
    }
    __syncthreads();
    if (threadIdx.x < D) {
        const int d = threadIdx.x;
        double* cd = cum + d * (bins + 1);
        double sum = 0.0;
        cd[0] = sum;
#pragma unroll 4
        for (int b = 0; b < bins; ++b) {
            sum += smooth[d * bins + b];
            cd[b + 1] = sum;
        }
    }
    __syncthreads();
    // every new edge finds its interval by itself (a forward walk of one thread per dimension
    // was a chain of dependent loads: 17 us for 32 bins, 33 us for 50)
    for (int t = threadIdx.x; t < D * (bins + 1); t += blockDim.x) {
        const int d = t / (bins + 1), k = t - d * (bins + 1);
        const double* cd = cum + d * (bins + 1);
        const double* e = edges + d * (bins + 1);
        const double total = cd[bins];
        const double step = total / bins;
        // torch.linspace(0, total, bins + 1); searchsorted(cum, target, right) - 1
        const double target = k < (bins + 1) / 2 ? step * k : total - step * (bins - k);
        int lo = 0, hi = bins;  // the number of j in 1..bins with cum[j] <= target
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (cd[mid + 1] <= target)
                lo = mid + 1;
            else
                hi = mid;
        }
        const int i = lo > bins - 1 ? bins - 1 : lo;
        const double frac = (target - cd[i]) / smooth[d * bins + i];
        next[t] = k == 0 ? 0.0 : k == bins ? 1.0 : e[i] + frac * (e[i + 1] - e[i]);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < D * (bins + 1); k += blockDim.x) edges[k] = next[k];
}

// One reported iteration of `samples` weights with sum s and sum of squares s2: its
// estimate and variance join the inverse-variance-weighted combination in the scalar slots
// sc; value, error and the convergence flag (after min_iterations, error <= max(epsabs,
// epsrel |value|)) are updated.  Returns the iteration's weight 1/variance.
__device__ inline double combine(double* sc, double s, double s2, double samples, int min_iterations, double epsrel,
                                 double epsabs)
{
    const double n = samples;
    const double est = s / n;
    double var = (s2 - s * s / n);
    var = var > 0.0 ? var : 0.0;
    var = var / (n - 1.0) / n;
    var = var > 2.2250738585072014e-308 ? var : 2.2250738585072014e-308;
    sc[kStSumWeightedEst] += est / var;
    sc[kStSumWeights] += 1.0 / var;
    sc[kStIterations] += 1.0;
    sc[kStLastEstimate] = est;
    sc[kStLastVariance] = var;
    const double value = sc[kStSumWeightedEst] / sc[kStSumWeights];
    const double error = ::sqrt(1.0 / sc[kStSumWeights]);
    sc[kStValue] = value;
    sc[kStError] = error;
    const double tol = epsabs > epsrel * ::fabs(value) ? epsabs : epsrel * ::fabs(value);
    if (sc[kStIterations] >= (double)min_iterations && error <= tol) sc[kStConverged] = 1.0;
    return 1.0 / var;
}

}  // namespace vegas
}  // namespace nlo
