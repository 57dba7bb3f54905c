// Right-hand-side assembly and the rapidity step (FP64).
//
// dN/dY = K1 + (K2+Kf) with non-finite values replaced by 0 (bk/evolution.py:329-351);
// inactive parents carry zeros because their K1 and K2+Kf entries are zeroed.
// A stage input is N + sum_k c_k k_k; the final combination of a step optionally
// clamps to [0,1] (FORCE_POSITIVE_N, bk/evolution.py:150-151) and flags
// non-finite values in a status word (bk/evolution.py:152-153 raises on the host).

#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"

namespace nlo {

namespace {

// dN/dY of one parent: K1 + (K2 + Kf), 0 where it is not finite.
__device__ __forceinline__ double assembled(double k1, const double* __restrict__ sums, double factor, double& nlo)
{
    nlo = (sums[0] + sums[1]) * factor;
    const double v = k1 + nlo;
    return isfinite(v) ? v : 0.0;
}

__global__ void assemble_kernel(const double* __restrict__ k1, const double* __restrict__ k2kf, int n,
                                double inv_samples, double* __restrict__ dndy, double* __restrict__ k2kf_total)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double nlo;
    dndy[i] = assembled(k1[i], k2kf + 3 * (size_t)i, inv_samples, nlo);
    if (k2kf_total) k2kf_total[i] = nlo;
}

struct StageArgs {
    const double* k[4];
    double c[4];
    int nk;
};

__device__ __forceinline__ double combined(double v, const StageArgs& a, size_t at, int clamp, uint32_t* status)
{
    for (int j = 0; j < a.nk; ++j) v += a.c[j] * a.k[j][at];
    if (clamp) v = v < 0.0 ? 0.0 : (v > 1.0 ? 1.0 : v);
    if (status && !isfinite(v)) atomicOr(status, (uint32_t)kStatusNonFinite);
    return v;
}

__global__ void axpy_stage_kernel(const double* N, StageArgs a, int n, double* out, int clamp,
                                  uint32_t* __restrict__ status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = combined(N[i], a, i, clamp, status);
}

// Several parameter sets (blockIdx.y): the end of a stage in one launch, the derivative of each parent
// and then the stage combination, whose terms read this thread's element only (the last of them
// just written).
__global__ void finish_stage_sets_kernel(const double* __restrict__ k1, const double* __restrict__ k2kf,
                                         const SetTable* __restrict__ table, double* dndy, RowsArg N, StageArgs a,
                                         int n, RowsArg out, int clamp, uint32_t* __restrict__ status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (i >= n) return;
    const size_t at = (size_t)s * n + i;
    double nlo;
    dndy[at] = assembled(k1[at], k2kf + 3 * at, table->inv[s], nlo);
    out.at(s)[i] = combined(N.at(s)[i], a, at, clamp, status ? status + s : nullptr);
}

__global__ void axpy_sets_kernel(RowsArg N, StageArgs a, int n, RowsArg out, int clamp, uint32_t* __restrict__ status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (i >= n) return;
    out.at(s)[i] = combined(N.at(s)[i], a, (size_t)s * n + i, clamp, status ? status + s : nullptr);
}

struct SetupArg {
    double* rows[kMaxSets];
    uint32_t samples[kMaxSets];
    uint16_t cta_first[kMaxSets + 1];
    int sets, nlo;
};
static_assert(sizeof(SetupArg) <= 4096, "the set table travels as a kernel parameter");

// Sobol directions of up to kDirsPerLaunch sets per launch (a large kernel parameter).
constexpr int kDirsPerLaunch = 48;
struct DirsArg {
    int first, count;
    uint32_t words[kDirsPerLaunch][kSetDirsWords];
};
static_assert(sizeof(DirsArg) <= 32000, "within the kernel parameter limit of sm_70 and later");

__global__ void sets_dirs_kernel(DirsArg a, SetTable* __restrict__ t)
{
    for (int i = threadIdx.x; i < a.count * kSetDirsWords; i += blockDim.x)
        t->dirs[a.first + i / kSetDirsWords][i % kSetDirsWords] = a.words[i / kSetDirsWords][i % kSetDirsWords];
}

__global__ void sets_setup_kernel(SetupArg a, SetTable* __restrict__ t)
{
    const int i = threadIdx.x;
    if (i < kMaxSets) {
        t->rows[i] = i < a.sets ? a.rows[i] : nullptr;
        t->samples[i] = i < a.sets ? a.samples[i] : 0u;
        t->inv[i] = i < a.sets && a.nlo && a.samples[i] > 0 ? 1.0 / (double)a.samples[i] : 0.0;
    }
    if (i <= a.sets) t->cta_first[i] = a.cta_first[i];
}

}  // namespace

cudaError_t launch_sets_setup(double* const* rows, const int64_t* samples, const uint16_t* cta_first,
                              const SobolDirsArg* const* dirs, int sets, bool nlo, SetTable* table,
                              cudaStream_t stream)
{
    if (sets < 1 || sets > kMaxSets) return cudaErrorInvalidValue;
    SetupArg a;
    for (int i = 0; i < kMaxSets; ++i) {
        a.rows[i] = i < sets ? rows[i] : nullptr;
        a.samples[i] = i < sets ? (uint32_t)samples[i] : 0u;
    }
    for (int i = 0; i <= kMaxSets; ++i) a.cta_first[i] = i <= sets ? cta_first[i] : (uint16_t)0;
    a.sets = sets;
    a.nlo = nlo ? 1 : 0;
    sets_setup_kernel<<<1, kMaxSets + 32, 0, stream>>>(a, table);
    cudaError_t e = cudaGetLastError();
    for (int first = 0; first < sets && e == cudaSuccess; first += kDirsPerLaunch) {
        DirsArg d;
        d.first = first;
        d.count = sets - first < kDirsPerLaunch ? sets - first : kDirsPerLaunch;
        for (int k = 0; k < d.count; ++k) {
            const SobolDirsArg& src = *dirs[first + k];
            for (int j = 0; j < 4; ++j) {
                for (int b = 0; b < 30; ++b) d.words[k][30 * j + b] = src.state[j][b];
                d.words[k][120 + j] = src.shift[j];
            }
        }
        sets_dirs_kernel<<<1, 256, 0, stream>>>(d, table);
        e = cudaGetLastError();
    }
    return e;
}

static StageArgs stage_args(const double* const* k, const double* coef, int nk)
{
    StageArgs a;
    a.nk = nk;
    for (int j = 0; j < 4; ++j) {
        a.k[j] = j < nk ? k[j] : nullptr;
        a.c[j] = j < nk ? coef[j] : 0.0;
    }
    return a;
}

cudaError_t launch_finish_stage_sets(const double* k1, const double* k2kf, const SetTable* table, double* dndy,
                                     const RowsArg& N, const double* const* k, const double* coef, int nk, int points,
                                     int sets, const RowsArg& out, int clamp, uint32_t* status, cudaStream_t stream)
{
    finish_stage_sets_kernel<<<dim3((points + 255) / 256, sets), 256, 0, stream>>>(
        k1, k2kf, table, dndy, N, stage_args(k, coef, nk), points, out, clamp, status);
    return cudaGetLastError();
}

cudaError_t launch_axpy_sets(const RowsArg& N, const double* const* k, const double* coef, int nk, int points,
                             int sets, const RowsArg& out, int clamp, uint32_t* status, cudaStream_t stream)
{
    axpy_sets_kernel<<<dim3((points + 255) / 256, sets), 256, 0, stream>>>(N, stage_args(k, coef, nk), points, out,
                                                                           clamp, status);
    return cudaGetLastError();
}

cudaError_t launch_assemble(const double* k1, const double* k2kf, int points, double inv_samples, double* dndy,
                            double* k2kf_total, cudaStream_t stream)
{
    assemble_kernel<<<(points + 255) / 256, 256, 0, stream>>>(k1, k2kf, points, inv_samples, dndy, k2kf_total);
    return cudaGetLastError();
}

cudaError_t launch_axpy_stage(const double* N, const double* const* k, const double* coef, int nk, int points,
                              double* out, int clamp, uint32_t* status, cudaStream_t stream)
{
    axpy_stage_kernel<<<(points + 255) / 256, 256, 0, stream>>>(N, stage_args(k, coef, nk), points, out, clamp,
                                                                status);
    return cudaGetLastError();
}

}  // namespace nlo
