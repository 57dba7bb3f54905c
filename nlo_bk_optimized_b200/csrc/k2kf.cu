// K2 + Kf: the NLO part of the BK right-hand side, integrated by quasi-Monte Carlo
// over scrambled Sobol points of the box (log z, log z', theta_z, theta_z') of
// bk/derivatives.py:424-431, with the integrand _nlo_integrand x exp(2 log z + 2 log z')
// of bk/derivatives.py:322-335 and 490-612 (kernels bk_kernels/k2.py:8-39 and
// bk_kernels/kf.py:10-41, coupling at the smallest dipole, RC_NLO = SMALLEST_NLO).
//
// Work decomposition (B200): the points are the same for every parent r, and z,
// z', |z - z'|, their three spline values, the dipole factors of the daughter
// dipoles and the Jacobian do not depend on r.  Each CTA therefore stages a tile
// of samples (one per thread) in shared memory, and every lane then owns one
// active parent and sweeps the whole tile, reading the sample records as
// shared-memory broadcasts.  Per (sample, parent) only X, X', their two spline
// values, the kernels and the coupling remain.  In the mixed build lane sums are FP32
// over 32 samples, folded into FP64 per lane (the FP64 build: compensated sums per
// tile); per-CTA partials go to the caller's workspace and a second kernel adds them in
// a fixed order (deterministic).

#include <cuda_runtime.h>

#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "k2kf_integrand.cuh"
#include "sobol.cuh"

namespace nlo {

namespace {

using namespace k2;

constexpr int kFoldPairs = 16;

// Shared-memory bytes of the spline tables: the T-typed log S coefficients, the
// pre-scaled FP32 rows with their edge rows (FP32 build) and the knots.
template <typename T>
__host__ __device__ inline size_t k2_table_bytes(int n)
{
    const size_t b = sizeof(T) * 4 * (size_t)(n - 1) + (sizeof(T) == sizeof(float) ? sizeof(float4) * (size_t)(n + 1) : 0) +
                     sizeof(T) * (size_t)n;
    return (b + 15) & ~(size_t)15;
}

template <typename T, bool SYM, int COUPLING>
__global__ void __launch_bounds__(448, (sizeof(T) == 4 ? 2 : 1)) k2kf_kernel(Phys<T> ph, K2Box<T> box, SobolDirsArg dirs,
                                                    const double* __restrict__ r_grid, int n,
                                                    const double* __restrict__ spline,
                                                    const int32_t* __restrict__ active,
                                                    const int32_t* __restrict__ count, uint64_t offset,
                                                    uint64_t samples, int tile_samples, double* __restrict__ partial)
{
    const uint64_t tile = tile_samples;
    const uint64_t tiles = (samples + tile - 1) / tile;

    extern __shared__ __align__(16) unsigned char k2_smem[];
    K2Rec<T>* recs = reinterpret_cast<K2Rec<T>*>(k2_smem);  // [blockDim.x], 16-byte aligned rows
    // cs [n-1][4] natural units, cs2 [n+1] pre-scaled with edge rows (FP32 path), xs [n]
    T* cs = reinterpret_cast<T*>(recs + blockDim.x);
    float4* cs2 = reinterpret_cast<float4*>(cs + 4 * (n - 1));
    T* xs = reinterpret_cast<T*>(cs2 + (sizeof(T) == sizeof(float) ? n + 1 : 0));
    uint32_t* st = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(cs) + k2_table_bytes<T>(n));  // [4][30] + shift[4]
    const double h64 = (spline[n - 1] - spline[0]) / (double)(n - 1);
    const double* src_coef = spline + n + 4 * (size_t)(n - 1);  // log S block
    for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = (T)spline[i];
    for (int i = threadIdx.x; i < 4 * (n - 1); i += blockDim.x) cs[i] = (T)src_coef[i];
    if constexpr (sizeof(T) == sizeof(float)) stage_fast_rows(cs2, src_coef, n, h64);
    for (int i = threadIdx.x; i < 120; i += blockDim.x) st[i] = dirs.state[i / 30][i % 30];
    if (threadIdx.x < 4) st[120 + threadIdx.x] = dirs.shift[threadIdx.x];
    __syncthreads();
    SplineView<T> s;
    s.x = xs;
    s.coef = cs;
    s.n = n;
    s.x0 = s.x[0];
    s.inv_h = (T)((double)(n - 1) / (spline[n - 1] - spline[0]));

    // per-evaluation spline: uniform-grid FP32 form in the mixed build, the exact
    // knot search in the FP64 build
    FastSpline fs;
    fs.coef = cs2;
    fs.u_scale = (float)(0.5 * 0.69314718055994531 / h64);
    fs.u_off = (float)(-spline[0] / h64);
    fs.u_top = (float)(n - 1);

    const int n_active = *count;
    const int slot = blockIdx.y * blockDim.x + threadIdx.x;
    const bool has_parent = slot < n_active;
    K2Parent<T> P;
    K2ParentF PF;
    {
        const double r = has_parent ? r_grid[active[slot]] : 1.0;
        P.r = (T)r;
        P.r2 = P.r * P.r;
        P.lr = (T)log(r);
        P.two_r = (T)2 * P.r;
        PF.r = (float)r;
        PF.r2 = (float)(r * r);
        PF.lr = (float)log(r);
        PF.two_r = (float)(2.0 * r);
        PF.four_r = (float)(4.0 * r);
        P.alpha_r = alpha_of_log(P.lr, ph);
        PF.alpha_r = (float)P.alpha_r;
    }
    double acc_k2 = 0.0, acc_kf = 0.0, acc_sq = 0.0;
    // CTAs whose parent tile is empty still stage samples for nobody: skip them.
    if (blockIdx.y * blockDim.x < (unsigned)n_active) {
        for (uint64_t tix = blockIdx.x; tix < tiles; tix += gridDim.x) {
            const uint64_t local = tix * tile + threadIdx.x;
            const uint64_t remaining = samples - tix * tile;
            const int count_here = (int)(remaining < tile ? remaining : tile);
            if constexpr (sizeof(T) == sizeof(float)) {
                // pair layout: the fields of samples 2p and 2p+1 side by side (the tile is even;
                // a padding sample past the budget carries zero weight)
                float rec[kRecLen];
                if (threadIdx.x < tile) {
                    k2_prepare<float>(s, box, st, st + 120, offset + local, local < samples, rec);
                    float* dst = reinterpret_cast<float*>(recs) + (size_t)(threadIdx.x >> 1) * (2 * kRecLen) +
                                 (threadIdx.x & 1);
#pragma unroll
                    for (int f = 0; f < kRecLen; ++f) dst[2 * f] = rec[f];
                }
                __syncthreads();
                if (has_parent) {
                    const float4* pr = reinterpret_cast<const float4*>(recs);
                    f2 sq = bc2(0.0f);  // variance estimate only: plain sum per tile
                    const int pairs = (count_here + 1) >> 1;
                    // FP32x2 partial sums of 16 pairs (32 samples), folded into FP64: the
                    // rounding of a 32-term FP32 sum instead of compensated summation.  The
                    // sums are of K2 + Kf and of Kf (K2 is their difference, formed once at
                    // the end): the total is needed anyway for the variance, and this saves
                    // the finite-test select of K2 per sample
                    for (int j0 = 0; j0 < pairs; j0 += kFoldPairs) {
                        const int jn = j0 + kFoldPairs < pairs ? j0 + kFoldPairs : pairs;
                        f2 ptot = bc2(0.0f), pkf = bc2(0.0f);
                        for (int j = j0; j < jn; ++j) {
                            f2 kfw, tot;
                            k2_pair_fast<SYM, COUPLING>(fs, ph, PF, pr + (kRecLen / 2) * j, kfw, tot);
                            ptot = add2(ptot, tot);
                            pkf = add2(pkf, kfw);
                            sq = fma2(tot, tot, sq);
                        }
                        acc_k2 += (double)ptot.x + (double)ptot.y;  // K2 + Kf until the end
                        acc_kf += (double)pkf.x + (double)pkf.y;
                    }
                    acc_sq += (double)sq.x + (double)sq.y;
                }
            } else {
                if (threadIdx.x < tile)
                    k2_prepare<T>(s, box, st, st + 120, offset + local, local < samples, recs[threadIdx.x].v);
                __syncthreads();
                if (has_parent) {
                    Kahan<T> sk2, skf;
                    sk2.reset();
                    skf.reset();
                    T sq = (T)0;  // variance estimate only: plain sum per tile
                    for (int j = 0; j < count_here; ++j) {
                        T k2w, kfw;
                        k2_point<T, SYM>(s, ph, P, recs[j].v, k2w, kfw);
                        sk2.add(k2w);
                        skf.add(kfw);
                        const T tot = k2w + kfw;
                        sq += tot * tot;
                    }
                    acc_k2 += (double)sk2.sum - (double)sk2.comp;
                    acc_kf += (double)skf.sum - (double)skf.comp;
                    acc_sq += (double)sq;
                }
            }
            __syncthreads();
        }
    }
    if (slot < n) {
        double* o = partial + ((size_t)blockIdx.x * n + slot) * 3;
        o[0] = sizeof(T) == sizeof(float) ? acc_k2 - acc_kf : acc_k2;
        o[1] = acc_kf;
        o[2] = acc_sq;
    }
}

// One warp per active parent: lanes add strided CTA partials, then a fixed
// shuffle tree combines them (the order does not depend on timing).
__global__ void __launch_bounds__(256) k2kf_finalize_kernel(const double* __restrict__ partial, int blocks, int n,
                                                            const int32_t* __restrict__ active,
                                                            const int32_t* __restrict__ count,
                                                            double* __restrict__ out)
{
    const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (slot >= n || slot >= *count) return;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int c = lane; c < blocks; c += 32) {
        const double* p = partial + ((size_t)c * n + slot) * 3;
        s0 += p[0];
        s1 += p[1];
        s2 += p[2];
    }
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, o);
        s1 += __shfl_down_sync(0xffffffffu, s1, o);
        s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        double* o = out + 3 * (size_t)active[slot];
        o[0] = s0;
        o[1] = s1;
        o[2] = s2;
    }
}

template <typename T>
size_t k2_smem_bytes(int threads, int points)
{
    return sizeof(K2Rec<T>) * threads + k2_table_bytes<T>(points) + sizeof(uint32_t) * kSetDirsWords;
}

template <typename T, bool SYM, int COUPLING>
cudaError_t launch_typed(const nlo_bk_params& p, const double* r, int points, const double* spline,
                         const int32_t* active, const int32_t* count, const SobolDirsArg& dirs, uint64_t offset,
                         uint64_t samples, const nlo_bk_box& box, double* partial, int max_blocks, int threads,
                         int parent_tiles, int* used_blocks, cudaStream_t stream)
{
    const size_t smem = k2_smem_bytes<T>(threads, points);
    cudaError_t e = raise_dynamic_smem((const void*)k2kf_kernel<T, SYM, COUPLING>, smem);
    if (e == cudaSuccess) e = prefer_shared_carveout((const void*)k2kf_kernel<T, SYM, COUPLING>);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k2kf_kernel<T, SYM, COUPLING>, threads, smem);
    if (e != cudaSuccess) return e;
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (per_sm < 1) per_sm = 1;
    // A GPU's worth of CTAs for every parent tile, not for all of them together: the tiles are
    // filled in order, so at 449 to about 490 points the second is empty (the saturated parents are
    // not active) and its CTAs return at once, and beyond that it has few parents.  One RK4 step,
    // 2^18 samples: 450 points 5.1 -> 3.6 ms, 520 points 5.6 -> 4.5, 700 points 7.2 -> 6.8.
    uint64_t blocks = (uint64_t)per_sm * sms;
    if (blocks > (uint64_t)max_blocks) blocks = (uint64_t)max_blocks;
    // The tile (a multiple of the 32 samples of an FP32 partial sum, at most one sample per thread)
    // for which a CTA's share of the samples rounds up least, with 8 samples' worth of staging a
    // tile: whole tiles of 416 gave 2^20 samples over 296 CTAs 8 tiles for some and 9 for others
    // (3,744 samples' time; 14 tiles of 256 are 3,584), and 2^14 samples at 200 parents 74 CTAs
    // with one tile of 224 each (512 of 32).
    const uint64_t share = (samples + blocks - 1) / blocks;
    uint64_t tile = (uint64_t)threads, best = ~(uint64_t)0;
    for (uint64_t t = 32; t <= (uint64_t)threads; t += 32) {
        const uint64_t cost = (share + t - 1) / t * (t + 8);
        if (cost <= best) {
            best = cost;
            tile = t;
        }
    }
    const uint64_t tiles = (samples + tile - 1) / tile;
    if (blocks > tiles) blocks = tiles;
    *used_blocks = (int)blocks;
    dim3 grid((unsigned)blocks, (unsigned)parent_tiles);
    k2kf_kernel<T, SYM, COUPLING><<<grid, threads, smem, stream>>>(
        make_phys<T>(p), make_box<T>(p, box, SYM), dirs, r, points, spline, active, count, offset, samples, (int)tile,
        partial);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_k2kf(const nlo_bk_params& p, const double* r, int points, const double* spline,
                        const int32_t* active, const int32_t* count, const SobolDirsArg& dirs, uint64_t offset,
                        uint64_t samples, const nlo_bk_box& box, double* out, double* partial, int max_blocks,
                        cudaStream_t stream, bool cleared)
{
    cudaError_t e = cleared ? cudaSuccess : cudaMemsetAsync(out, 0, sizeof(double) * 3 * (size_t)points, stream);
    if (e != cudaSuccess || samples == 0) return e;
    // 448 threads, two CTAs per SM: 72 registers without spills
    int threads = ((points < kLaneCap ? points : kLaneCap) + 31) / 32 * 32;
    if (threads < 64) threads = 64;
    const int parent_tiles = (points + threads - 1) / threads;
    int used = 0;
    e = dispatch_variant(p, [&](auto t, auto sym, auto c) {
        return launch_typed<decltype(t), decltype(sym)::value, decltype(c)::value>(
            p, r, points, spline, active, count, dirs, offset, samples, box, partial, max_blocks, threads, parent_tiles,
            &used, stream);
    });
    if (e != cudaSuccess) return e;
    k2kf_finalize_kernel<<<(points * 32 + 255) / 256, 256, 0, stream>>>(partial, used, points, active, count, out);
    return cudaGetLastError();
}

}  // namespace nlo
