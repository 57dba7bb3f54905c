// K2 + Kf by Vegas: the reference's default integrator for the NLO part of the BK
// right-hand side (rapidity_derivative_nlo with IntegrationMethod.VEGAS,
// bk/derivatives.py:389-421 -- 32 bins, a warm-up of max(2, MCINTPOINTS/5) samples, at
// least 2 and at most 4 iterations, epsrel 0.2 -- driving vegas(), numerics/integration.py:
// 120-589), with each parent's importance grid carried from one right-hand side to the next
// and refreshed by a shortened warm-up (VEGAS_REUSE_GRID, VEGAS_REUSE_WARMUP_FRACTION; the
// per-parent vegas_states of bk/evolution.py:85-100 and 354-424).
//
// Every active parent is one integral with its own grid; all of them run in the same
// launches.  A round (the warm-up, or one iteration) is two launches: the round kernel
// (grid: CTAs per parent x integrals) maps scrambled Sobol points through the parent's
// grid, evaluates the full integrand and leaves per-CTA sums of w, w^2, w_K2, w_Kf and the
// |w| histograms; a finalize CTA per integral adds them in a fixed order, re-bins the grid
// and folds the iteration into the inverse-variance combination (vegas_common.cuh, the code
// the DIS terms use).  Converged parents skip the remaining rounds, so the host enqueues
// every round without synchronising.
//
// Samples: the Sobol points of `dirs`, indices 0, 1, ... across the rounds of one
// right-hand side (the warm-up first); every parent and every right-hand side starts again
// at index 0, as the reference restarts its generator from the same seed in every vegas()
// call.  A coordinate u gives the bin floor(u bins) and the fraction u bins - bin.
#include <cuda_runtime.h>

#include <cstring>

#include "common.cuh"
#include "internal.h"
#include "k2kf_integrand.cuh"
#include "sobol.cuh"
#include "vegas_common.cuh"
#include "vegas_sampling.cuh"

namespace nlo {

namespace {

using namespace k2;
using namespace vegas;

constexpr int kDims = 4;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// BK slots after the generic ones of vegas_common.cuh (all < kStSlots)
enum BkSlot {
    kBkHasGrid = 9,   // the grid was adapted by an earlier right-hand side (persistent)
    kBkWarmup = 10,   // warm-up samples of this right-hand side
    kBkOffset = 11,   // Sobol index of the next round
    kBkActive = 12,   // the parent is integrated in this right-hand side
    kBkCompK2 = 13,   // sum over iterations of weight x K2 estimate
    kBkCompKf = 14,   // sum over iterations of weight x Kf estimate
};

// Per-parent accumulators of the replica refinement: [selected, sum of values, sum of error^2].
constexpr int kRepStride = 3;

__device__ __forceinline__ bool parent_active(const double* N, int i, int shard, int shards)
{
    return i > 0 && N[i] <= 0.99999 && i % shards == shard;
}

// Per integral: mark whether it is taken, reset the per-call sums, and either start a uniform
// grid with the full warm-up or keep the stored grid with the reuse warm-up.  Integral
// blockIdx.x is parent blockIdx.x % points.  select (replica rounds): the parents to integrate
// are those with select[parent * kRepStride] != 0.
__global__ void begin_kernel(const double* __restrict__ N, int points, int shard, int shards, double* state,
                             int stride, int bins, int reuse, uint64_t warmup, uint64_t reuse_warmup,
                             int32_t* __restrict__ counts, const double* __restrict__ select)
{
    const int i = blockIdx.x;
    const int parent = i % points;
    double* st = state + (size_t)i * stride;
    double* sc = st + kDims * (bins + 1);
    const bool on = select ? select[(size_t)parent * kRepStride] != 0.0 : parent_active(N, parent, shard, shards);
    __syncthreads();
    const bool fresh = !reuse || sc[kBkHasGrid] == 0.0;
    if (on) {
        for (int k = threadIdx.x; k < kDims * bins; k += blockDim.x) counts[(size_t)i * kDims * bins + k] = 0;
        if (fresh)
            for (int k = threadIdx.x; k < kDims * (bins + 1); k += blockDim.x) {
                const int b = k % (bins + 1);
                st[k] = b == bins ? 1.0 : (double)b / bins;
            }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (on) {
            for (int k = 0; k <= kStLastVariance; ++k) sc[k] = 0.0;
            sc[kBkCompK2] = 0.0;
            sc[kBkCompKf] = 0.0;
            sc[kBkWarmup] = (double)(fresh ? warmup : reuse_warmup);
            sc[kBkOffset] = 0.0;
        }
        sc[kBkActive] = on ? 1.0 : 0.0;
    }
}

// Direction numbers of the integrals of one launch: set 0 of the main integrals, set g of the
// g-th replica (integral / points).
constexpr int kReplicaSets = 16;  // options.replicas is at most 16
struct BkDirs {
    uint32_t state[kReplicaSets][kDims][30];
    uint32_t shift[kReplicaSets][kDims];
};

// Samples of parent slot `sc` in this round (0: skip the parent).
__device__ __forceinline__ uint64_t round_samples(const double* sc, int warmup, uint64_t samples)
{
    if (sc[kBkActive] == 0.0 || sc[kStConverged] != 0.0) return 0;
    return warmup ? (uint64_t)sc[kBkWarmup] : samples;
}

// The FP32 build takes two blocks of 32 samples a pass on the packed FP32x2 instructions, with
// the QMC kernel's evaluation (k2_pair_fast) on a FineSpline and the record formed in registers; FP64
// takes one.  K2 and Kf are added, and their sums kept, in FP64.  What bounds it: instruction issue.
// BKConfig() to Y = 0.4 takes 15.8 ms, 24.3 with the scalar evaluation (k2_prepare_x, k2_point).
// Errors of one round against FP64 on the same points, norm over the parents, mean of 24 cases
// (50 to 200 points, 5,000 to 60,000 samples, both symmetrisations and couplings): 2.8e-6 on the
// uniform grid and 6.6e-6 on adapted ones; scalar 2.9e-6 and 1.5e-5.
template <typename T, bool SYM, int COUPLING>
__global__ void __launch_bounds__(kThreads, (sizeof(T) == 4 ? 3 : 2)) round_kernel(Phys<T> ph, K2Box<T> box,
                                                         const __grid_constant__ BkDirs dirs,
                                                         const double* __restrict__ r_grid, int n,
                                                         const double* __restrict__ spline, const double* state,
                                                         int stride, int bins, int warmup, uint64_t samples,
                                                         int blocks_per_job, double* __restrict__ partial,
                                                         int32_t* __restrict__ counts)
{
    const int job = blockIdx.y;
    const double* st = state + (size_t)job * stride;
    const double* sc = st + kDims * (bins + 1);
    const uint64_t total = round_samples(sc, warmup, samples);
    if (total == 0) return;  // uniform per CTA

    constexpr bool FAST = sizeof(T) == sizeof(float);
    extern __shared__ __align__(16) unsigned char vsm[];
    double2* cells = reinterpret_cast<double2*>(vsm);           // [4][bins] left end and 2^-30 width, box units
    double* density = reinterpret_cast<double*>(cells + kDims * bins);  // [4][bins] bins x width, unit cube
    double* whist = density + kDims * bins;                     // [warps][4*bins]
    int32_t* cnt = reinterpret_cast<int32_t*>(whist + kWarps * kDims * bins);  // [4*bins]
    unsigned char* tables = reinterpret_cast<unsigned char*>(cnt + kDims * bins);  // 16-byte aligned
    float4* rows = reinterpret_cast<float4*>(tables);           // FP32: [n+1] FastSpline rows
    double* xs = reinterpret_cast<double*>(tables);             // FP64: knots [n] ...
    double* cs = xs + ((n + 1) & ~1);                           // ... and the log S block [n-1][4]
    __shared__ SobolWarp<kDims> sobol;
    __shared__ double red[4][kWarps];

    const int set = job / n;
    const double* src_coef = spline + n + 4 * (size_t)(n - 1);
    const double fb = (double)bins;
    for (int k = threadIdx.x; k < kDims * bins; k += blockDim.x) {
        const int d = k / bins, e = k + d;
        const double left = st[e], width = st[e + 1] - left, span = (double)box.width[d];
        cells[k] = make_double2((double)box.lower[d] + span * left, span * width * 9.313225746154785e-10);
        density[k] = fb * width;
        cnt[k] = 0;
    }
    for (int k = threadIdx.x; k < kWarps * kDims * bins; k += blockDim.x) whist[k] = 0.0;
    const double h = (spline[n - 1] - spline[0]) / (double)(n - 1);
    if constexpr (FAST) {
        stage_fast_rows(rows, src_coef, n, h);
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = spline[i];
        for (int i = threadIdx.x; i < 4 * (n - 1); i += blockDim.x) cs[i] = src_coef[i];
    }
    stage_sobol(sobol, dirs.state[set], dirs.shift[set], bins);
    __syncthreads();

    const double r = r_grid[job - set * n];
    FineSpline fs;
    K2ParentF PF;
    SplineView<double> s;
    K2Parent<double> P;
    if constexpr (FAST) {
        fs = fine_spline(rows, n, spline[0], h);
        PF = fine_parent(r, ph);
    } else {
        s.x = xs;
        s.coef = cs;
        s.n = n;
        s.x0 = xs[0];
        s.inv_h = 1.0 / h;
        P.r = r;
        P.r2 = r * r;
        P.lr = log(r);
        P.two_r = 2.0 * r;
        P.alpha_r = alpha_of_log(P.lr, ph);
    }

    // this CTA's share of the round's Sobol indices [first, last), in blocks of 32 aligned indices
    const uint64_t first = (uint64_t)sc[kBkOffset], last = first + total;
    const uint64_t block0 = first >> 5, blocks = ((last + 31) >> 5) - block0;
    const uint64_t share = (blocks + blocks_per_job - 1) / blocks_per_job;
    const uint64_t begin = (uint64_t)blockIdx.x * share;
    const uint64_t end = begin + share < blocks ? begin + share : blocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* myhist = whist + warp * kDims * bins;
    double sw = 0.0, sw2 = 0.0, sk2 = 0.0, skf = 0.0;
    int whole = 0;
    // a block's point of this lane: box position, weight factor, where it falls
    struct Sample {
        uint32_t base, bits[kDims];
        int bin[kDims];
        T x[kDims];
        double factor;
        bool on;
    };
    auto sample = [&](uint64_t k, Sample& p) {
        p.base = (uint32_t)((block0 + k) << 5);
        const uint64_t index = (uint64_t)p.base + lane;
        p.on = k < end && index >= first && index < last;
        p.factor = 1.0;
#pragma unroll
        for (int d = 0; d < kDims; ++d) {
            p.bits[d] = sobol_block_bits(sobol, d, p.base);
            double rest;
            p.bin[d] = grid_position(p.bits[d], bins, rest);
            const double2 cell = cells[d * bins + p.bin[d]];
            p.x[d] = (T)fma(rest, cell.y, cell.x);
            p.factor *= density[d * bins + p.bin[d]];
        }
    };
    auto record = [&](const Sample& p, double k2_w, double kf_w) {
        // a lane without a sample adds zeros and no counts
        const double factor = p.on ? p.factor : 0.0;
        const double w = (k2_w + kf_w) * factor, wk2 = k2_w * factor, wkf = kf_w * factor;
        sw += w;
        sw2 += w * w;
        sk2 += wk2;
        skf += wkf;
        const double aw = ::fabs(w);
        warp_hist_add(sobol, p.base, p.bits, p.on, p.bin, bins, aw, myhist, cnt, whole);
    };
    for (uint64_t k = begin + warp; k < end; k += FAST ? 2 * kWarps : kWarps) {
        Sample a;
        sample(k, a);
        if constexpr (FAST) {
            Sample b;
            sample(k + kWarps, b);
            float4 rec4[kRecLen / 2];
            k2_prepare_pair(fs, box.cpt_scale, make_float2(a.x[0], b.x[0]), make_float2(a.x[1], b.x[1]),
                            make_float2(a.x[2], b.x[2]), make_float2(a.x[3], b.x[3]), rec4);
            f2 kf, k2;
            k2_pair_fast<SYM, COUPLING>(fs, ph, PF, rec4, kf, k2);
            record(a, (double)k2.x, (double)kf.x);
            record(b, (double)k2.y, (double)kf.y);
        } else {
            T rec[kRecLen];
            k2_prepare_x<T>(s, box, a.x, true, rec);
            T k2w, kfw;
            k2_point<T, SYM>(s, ph, P, rec, k2w, kfw);
            record(a, k2w, kfw);
        }
    }
    add_whole_blocks<kDims>(whole, cnt);
    for (int o = 16; o > 0; o >>= 1) {
        sw += __shfl_down_sync(0xffffffffu, sw, o);
        sw2 += __shfl_down_sync(0xffffffffu, sw2, o);
        sk2 += __shfl_down_sync(0xffffffffu, sk2, o);
        skf += __shfl_down_sync(0xffffffffu, skf, o);
    }
    if (lane == 0) {
        red[0][warp] = sw;
        red[1][warp] = sw2;
        red[2][warp] = sk2;
        red[3][warp] = skf;
    }
    __syncthreads();
    // partial row: [sum w, sum w^2, hist[4][bins], sum w_K2, sum w_Kf]
    const int keys = 4 + kDims * bins;
    double* out = partial + ((size_t)job * blocks_per_job + blockIdx.x) * keys;
    if (threadIdx.x == 0) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        for (int w = 0; w < kWarps; ++w)
            for (int q = 0; q < 4; ++q) a[q] += red[q][w];
        out[0] = a[0];
        out[1] = a[1];
        out[2 + kDims * bins] = a[2];
        out[3 + kDims * bins] = a[3];
    }
    int32_t* cout = counts + (size_t)job * kDims * bins;
    for (int k = threadIdx.x; k < kDims * bins; k += blockDim.x) {
        double h = 0.0;
        for (int w = 0; w < kWarps; ++w) h += whist[w * kDims * bins + k];
        out[2 + k] = h;
        if (cnt[k]) atomicAdd(&cout[k], cnt[k]);
    }
}

// Per integral: add the round's partial rows in a fixed order (four interleaved chains per
// key, then the chains), re-bin the grid from the histogram and, for an iteration, fold its
// estimate into the weighted combination (value, error, convergence) and the K2 / Kf
// components; then advance the Sobol offset.
constexpr int kFinalThreads = 544;  // 4 x (4 + 4 x 32) sums at the default 32 bins

__global__ void __launch_bounds__(kFinalThreads)
    finalize_kernel(double* state, int stride, int bins, int warmup, uint64_t samples,
                    const double* __restrict__ partial, int blocks_per_job, int32_t* __restrict__ counts,
                    int min_iterations, double epsrel, double epsabs)
{
    extern __shared__ double fsm[];
    const int keys = 4 + kDims * bins;
    double* red = fsm;                       // [keys]
    double* chain = red + keys;              // [4][keys], then the re-binning's scratch:
    double* smooth = chain;                  // [4*bins]
    double* cum = smooth + kDims * bins;     // [4*(bins+1)]
    double* next = cum + kDims * (bins + 1); // [4*(bins+1)]
    // the scalar slots in shared memory: one trip to L2 instead of one per dependent access
    __shared__ double sc[kStSlots];
    const int job = blockIdx.x;
    double* st = state + (size_t)job * stride;
    double* slots = st + kDims * (bins + 1);
    if (threadIdx.x < kStSlots) sc[threadIdx.x] = slots[threadIdx.x];
    __syncthreads();
    const uint64_t n_round = round_samples(sc, warmup, samples);
    if (n_round == 0) return;
    const double* rows = partial + (size_t)job * blocks_per_job * keys;
    for (int t = threadIdx.x; t < 4 * keys; t += blockDim.x) {
        const int q = t / keys, k = t - q * keys;
        double sum = 0.0;
#pragma unroll 8
        for (int b = q; b < blocks_per_job; b += 4) sum += rows[(size_t)b * keys + k];
        chain[t] = sum;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < keys; k += blockDim.x)
        red[k] = (chain[k] + chain[keys + k]) + (chain[2 * keys + k] + chain[3 * keys + k]);
    __syncthreads();
    int32_t* c = counts + (size_t)job * kDims * bins;
    // the last thread's chain of divisions runs beside the re-binning
    if (threadIdx.x == blockDim.x - 1) {
        const double n = (double)n_round;
        sc[kStEvals] += n;
        if (!warmup) {
            const double weight = combine(sc, red[0], red[1], n, min_iterations, epsrel, epsabs);
            sc[kBkCompK2] += weight * (red[2 + kDims * bins] / n);
            sc[kBkCompKf] += weight * (red[3 + kDims * bins] / n);
        }
        sc[kBkOffset] += n;
        sc[kBkHasGrid] = 1.0;
    }
    rebin(st, red + 2, c, kDims, bins, smooth, cum, next);
    __syncthreads();
    for (int k = threadIdx.x; k < kDims * bins; k += blockDim.x) c[k] = 0;
    __syncthreads();
    if (threadIdx.x < kStSlots) slots[threadIdx.x] = sc[threadIdx.x];
}

// The right-hand side's K2+Kf per parent in the layout of nlo_bk_k2kf's sums: [value, 0,
// error^2] (assembled with the factor 1), zeros for parents not integrated.
__global__ void end_kernel(const double* state, int stride, int bins, int points, double* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= points) return;
    const double* sc = state + (size_t)i * stride + kDims * (bins + 1);
    const bool on = sc[kBkActive] != 0.0;
    out[3 * i + 0] = on ? sc[kStValue] : 0.0;
    out[3 * i + 1] = 0.0;
    out[3 * i + 2] = on ? sc[kStError] * sc[kStError] : 0.0;
}

// Replica refinement of bk/evolution.py:411-456 (the reference's CUDA mixed evolution with
// per-parent grids): a parent whose K1 and combined K2, Kf estimates cancel strongly,
// (|K1| + |K2| + |Kf|) / max(|K1 + K2 + Kf|, 0.05 (|K1| + |K2| + |Kf|)) >= 4, or whose
// amplitude exceeds 0.9, gets `replicas` more Vegas integrals on fresh grids with the seeds
// seed + 1000 k, and its K2+Kf becomes the mean of all of them, with the error
// sqrt(sum error^2) / (replicas + 1).  The parent's own grid is kept.
__global__ void replica_select_kernel(const double* __restrict__ N, const double* __restrict__ k1, int points,
                                      const double* __restrict__ state, int stride, int bins,
                                      double* __restrict__ acc)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= points) return;
    const double* sc = state + (size_t)i * stride + kDims * (bins + 1);
    double* a = acc + (size_t)i * kRepStride;
    a[0] = 0.0;
    if (sc[kBkActive] == 0.0 || !(sc[kStSumWeights] > 0.0)) return;
    const double c2 = sc[kBkCompK2] / sc[kStSumWeights];
    const double cf = sc[kBkCompKf] / sc[kStSumWeights];
    const double scale = ::fabs(k1[i]) + ::fabs(c2) + ::fabs(cf);
    const double net = ::fabs(k1[i] + c2 + cf);
    const double condition = scale / (net > 0.05 * scale ? net : 0.05 * scale);
    if (condition >= 4.0 || N[i] > 0.9) {
        a[0] = 1.0;
        a[1] = sc[kStValue];
        a[2] = sc[kStError] * sc[kStError];
    }
}

// The sums of `group` replicas (integral = g * points + parent), in replica order.
__global__ void replica_add_kernel(const double* __restrict__ state, int stride, int bins, int points, int group,
                                   double* __restrict__ acc)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= points) return;
    double* a = acc + (size_t)i * kRepStride;
    if (a[0] == 0.0) return;
    for (int g = 0; g < group; ++g) {
        const double* sc = state + ((size_t)g * points + i) * stride + kDims * (bins + 1);
        a[1] += sc[kStValue];
        a[2] += sc[kStError] * sc[kStError];
    }
}

__global__ void replica_end_kernel(const double* __restrict__ acc, int points, int replicas, double* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= points) return;
    const double* a = acc + (size_t)i * kRepStride;
    if (a[0] == 0.0) return;
    const double m = (double)(replicas + 1);
    out[3 * i + 0] = a[1] / m;
    out[3 * i + 2] = a[2] / (m * m);
}

// CTAs per integral: about 2,048 samples each (eight passes of a CTA, enough to outweigh
// staging its tables: a lone unconverged parent then spreads over 49 SMs at 1e5 samples,
// where 18 CTAs took 140 us a round), within 16,384 partial rows in all.
int bk_vegas_blocks_per_job(int points, int64_t samples)
{
    const int64_t by_rows = points < 16384 ? 16384 / points : 1;
    const int64_t want = (samples + 2047) / 2048;
    const int64_t b = want < by_rows ? want : by_rows;
    return (int)(b < 1 ? 1 : (b > 64 ? 64 : b));
}

// One round over `group` sets of `points` integrals (the main ones, or a group of replicas).
struct RoundArgs {
    const nlo_bk_params& p;
    const double* r;
    int points, group;
    const double* spline;
    const nlo_bk_box& box;
    const BkVegasCall& call;
    double* state;
    int blocks_per_job;
    cudaStream_t stream;
};

template <typename T, bool SYM, int COUPLING>
cudaError_t launch_round(const RoundArgs& a, const BkDirs& dirs, int warmup, int blocks)
{
    const int bins = a.call.options.bins;
    const size_t tables = sizeof(T) == sizeof(float) ? sizeof(float4) * (size_t)(a.points + 1)
                                                     : sizeof(double) * (size_t)(((a.points + 1) & ~1) + 4 * (a.points - 1));
    const size_t smem = (sizeof(double2) + sizeof(double) * (1 + kWarps) + sizeof(int32_t)) * kDims * (size_t)bins + tables;
    auto kern = round_kernel<T, SYM, COUPLING>;
    cudaError_t e = raise_dynamic_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    K2Box<T> kb;
    for (int d = 0; d < 4; ++d) {
        kb.lower[d] = (T)a.box.lower[d];
        kb.width[d] = (T)a.box.width[d];
    }
    const double volume = a.box.width[0] * a.box.width[1] * a.box.width[2] * a.box.width[3];
    // k2_pair_fast expects the symmetrisation's 1/2 in the weight
    const double half = sizeof(T) == sizeof(float) && SYM ? 0.5 : 1.0;
    kb.cpt_scale = (T)(half * volume * a.p.nc * a.p.nc / (8.0 * kPi * kPi * kPi * kPi));
    dim3 grid((unsigned)blocks, (unsigned)(a.points * a.group));
    kern<<<grid, kThreads, smem, a.stream>>>(make_phys<T>(a.p), kb, dirs, a.r, a.points, a.spline, a.state,
                                             a.call.stride, bins, warmup,
                                             (uint64_t)a.call.options.samples_per_iteration, blocks, a.call.partial,
                                             a.call.counts);
    return cudaGetLastError();
}

// The warm-up round (when `with_warmup`) and the iterations of one Vegas call over the
// integrals that the state marks active; `dirs`: the direction numbers of the a.group sets.
cudaError_t run_rounds(const RoundArgs& a, const SobolDirsArg* dirs, bool with_warmup)
{
    const nlo_bk_vegas_options& o = a.call.options;
    BkDirs sets;
    std::memset(&sets, 0, sizeof(sets));
    for (int g = 0; g < a.group; ++g) {
        std::memcpy(sets.state[g], dirs[g].state, sizeof(sets.state[g]));
        std::memcpy(sets.shift[g], dirs[g].shift, sizeof(sets.shift[g]));
    }
    const int keys = 4 + kDims * o.bins;
    const size_t fsmem = sizeof(double) * 5 * (size_t)keys;
    cudaError_t e = raise_dynamic_smem((const void*)finalize_kernel, fsmem);
    if (e != cudaSuccess) return e;
    const int rounds = o.max_iterations + (with_warmup ? 1 : 0);
    for (int k = 0; k < rounds; ++k) {
        const int warmup = with_warmup && k == 0;
        // a round of fewer samples (the warm-up) takes fewer CTAs per integral
        const int64_t n = warmup ? o.warmup_samples : o.samples_per_iteration;
        const int wanted = bk_vegas_blocks_per_job(a.points, n);
        const int blocks = wanted < a.blocks_per_job ? wanted : a.blocks_per_job;
        e = dispatch_variant(a.p, [&](auto t, auto sym, auto c) {
            return launch_round<decltype(t), decltype(sym)::value, decltype(c)::value>(a, sets, warmup, blocks);
        });
        if (e != cudaSuccess) return e;
        finalize_kernel<<<a.points * a.group, kFinalThreads, fsmem, a.stream>>>(
            a.state, a.call.stride, o.bins, warmup, (uint64_t)o.samples_per_iteration, a.call.partial, blocks,
            a.call.counts, o.min_iterations, o.epsrel, o.epsabs);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Integrals of one launch at most: replicas run together up to this many, at least one replica
// of every parent.
constexpr int kJobsCap = 4096;
}  // namespace

size_t bk_vegas_state_doubles(int bins) { return (size_t)kDims * (bins + 1) + kStSlots; }

int bk_vegas_replica_group(int points, int replicas)
{
    const int fit = kJobsCap / points;
    const int g = fit < replicas ? fit : replicas;
    return g < 1 ? 1 : g;
}

// A replica round has a few parents of each replica: half the CTAs of a main integral.
static int replica_blocks(int blocks) { return blocks > 1 ? blocks / 2 : 1; }

static size_t partial_rows(int points, const nlo_bk_vegas_options& o)
{
    const int64_t most = o.samples_per_iteration > o.warmup_samples ? o.samples_per_iteration : o.warmup_samples;
    const int blocks = bk_vegas_blocks_per_job(points, most);
    const size_t main = (size_t)points * blocks;
    const size_t rep = (size_t)points * bk_vegas_replica_group(points, o.replicas) * replica_blocks(blocks);
    return o.replicas > 0 && rep > main ? rep : main;
}

size_t bk_vegas_scratch_bytes(int points, const nlo_bk_vegas_options& o)
{
    const size_t keys = 4 + (size_t)kDims * o.bins;
    const size_t jobs = (size_t)points * bk_vegas_replica_group(points, o.replicas);
    // round partials, bin counts, then the replica grids and accumulators
    return sizeof(double) * keys * partial_rows(points, o) + sizeof(int32_t) * (size_t)kDims * o.bins * jobs + 256 +
           sizeof(double) * (bk_vegas_state_doubles(o.bins) * jobs + kRepStride * (size_t)points) + 256;
}

BkVegasCall bk_vegas_carve(void* scratch, int points, const nlo_bk_vegas_options& options, double* state)
{
    BkVegasCall c;
    c.options = options;
    c.state = state;
    c.stride = (int)bk_vegas_state_doubles(options.bins);
    const int64_t most = options.samples_per_iteration > options.warmup_samples ? options.samples_per_iteration
                                                                                : options.warmup_samples;
    c.blocks_per_job = bk_vegas_blocks_per_job(points, most);
    const size_t keys = 4 + (size_t)kDims * options.bins;
    const size_t jobs = (size_t)points * bk_vegas_replica_group(points, options.replicas);
    char* base = static_cast<char*>(scratch);
    c.partial = reinterpret_cast<double*>(base);
    c.counts = reinterpret_cast<int32_t*>(c.partial + keys * partial_rows(points, options));
    const size_t after = reinterpret_cast<size_t>(c.counts + (size_t)kDims * options.bins * jobs);
    c.replica_state = reinterpret_cast<double*>((after + 255) & ~(size_t)255);
    c.replica_acc = c.replica_state + bk_vegas_state_doubles(options.bins) * jobs;
    return c;
}

cudaError_t launch_k2kf_vegas(const nlo_bk_params& p, const double* r, const double* N, int points,
                              const double* spline, int shard, int shards, const SobolDirsArg& dirs,
                              const nlo_bk_box& box, const BkVegasCall& call, double* out, cudaStream_t stream)
{
    const nlo_bk_vegas_options& o = call.options;
    const uint64_t warmup = (uint64_t)o.warmup_samples;
    // numerics/integration.py:207-213: a reused grid is refreshed by max(2, warmup x fraction)
    // samples, or none when the warm-up or the fraction is zero
    uint64_t reuse_warmup = 0;
    if (warmup > 0 && o.reuse_warmup_fraction > 0.0) {
        reuse_warmup = (uint64_t)((double)warmup * o.reuse_warmup_fraction);
        if (reuse_warmup < 2) reuse_warmup = 2;
    }
    begin_kernel<<<points, 64, 0, stream>>>(N, points, shard, shards, call.state, call.stride, o.bins,
                                             o.reuse_grid ? 1 : 0, warmup, reuse_warmup, call.counts, nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const RoundArgs rounds{p, r, points, 1, spline, box, call, call.state, call.blocks_per_job, stream};
    if ((e = run_rounds(rounds, &dirs, warmup > 0 || reuse_warmup > 0)) != cudaSuccess) return e;
    end_kernel<<<(points + 255) / 256, 256, 0, stream>>>(call.state, call.stride, o.bins, points, out);
    return cudaGetLastError();
}

cudaError_t launch_k2kf_vegas_refine(const nlo_bk_params& p, const double* r, const double* N, int points,
                                     const double* spline, const nlo_bk_box& box, const BkVegasCall& call,
                                     const double* k1, double* out, cudaStream_t stream)
{
    const nlo_bk_vegas_options& o = call.options;
    if (o.replicas <= 0) return cudaSuccess;
    const int threads = 128, blocks = (points + threads - 1) / threads;
    replica_select_kernel<<<blocks, threads, 0, stream>>>(N, k1, points, call.state, call.stride, o.bins,
                                                          call.replica_acc);
    cudaError_t e = cudaGetLastError();
    // each replica: a fresh grid with the full warm-up (the reference's new VegasState); the
    // replicas are independent, so a group of them shares its launches (one by one, each left
    // most SMs idle: a typical right-hand side refines 17 of 92 parents)
    const uint64_t warmup = (uint64_t)o.warmup_samples;
    const int group = bk_vegas_replica_group(points, o.replicas);
    for (int k = 0; k < o.replicas && e == cudaSuccess; k += group) {
        const int sets = k + group <= o.replicas ? group : o.replicas - k;
        begin_kernel<<<points * sets, 64, 0, stream>>>(N, points, 0, 1, call.replica_state, call.stride, o.bins, 0,
                                                        warmup, 0, call.counts, call.replica_acc);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        const RoundArgs rounds{p,    r,
                               points, sets,
                               spline, box,
                               call,   call.replica_state,
                               replica_blocks(call.blocks_per_job), stream};
        if ((e = run_rounds(rounds, call.replica_dirs + k, warmup > 0)) != cudaSuccess) break;
        replica_add_kernel<<<blocks, threads, 0, stream>>>(call.replica_state, call.stride, o.bins, points, sets,
                                                           call.replica_acc);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    replica_end_kernel<<<blocks, threads, 0, stream>>>(call.replica_acc, points, o.replicas, out);
    return cudaGetLastError();
}

}  // namespace nlo
