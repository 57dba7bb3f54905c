// K2 + Kf of several parameter sets in one launch: the integrand and the fixed Sobol points of the
// one-set kernel (k2kf.cu; bk/derivatives.py:322-335, 424-431 and 490-612), each set with its own
// amplitudes, active points, budget and directions.
//
// Work decomposition (B200): a CTA of 8 warps belongs to one set and owns a contiguous range of its
// 32-sample chunks; the sets get CTAs in proportion to their budgets.  The CTA stages up to 8
// chunks of sample records (one per thread) in shared memory, and its warps sweep them for every
// active parent, one parent per lane, reading the records as shared-memory broadcasts.  The
// (32 parents, chunk) units of a tile go to the warps in equal contiguous shares: however many
// parents a set has, no warp waits at a barrier for more than one unit of another, and three CTAs
// fill an SM with two warps of each per scheduler.  Sums are those of the one-set kernel (FP32 over
// a chunk, folded into FP64), kept per (warp, group) in shared memory and added in warp order;
// per-CTA partials go to the workspace and a second kernel adds them in a fixed order.
//
// What bounds it: instruction issue and the MUFU pipe.  24 sets of 200 points with budgets of 2^16
// to 2^18: two RK4 steps in 36.6 ms, 39.3 with two sets to a CTA of 448 lanes (a set's last group
// of 32 and its shorter budget left lanes and warps idle at the barriers; the rate was 1.84e11
// evaluations/s).  One set over the whole GPU (400 points, 2^20 samples, RK4) is 4 % faster with a
// warp per 32 parents (k2kf.cu: 26 warps of 72 registers per SM, 24 of 80 here; this form at 28
// warps of 72 spills and took 16 % longer), so that form stays for one set.

#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"
#include "k2kf_integrand.cuh"
#include "sobol.cuh"

namespace nlo {

namespace {

using namespace k2;

constexpr int kK2Warps = 8;
constexpr int kK2Threads = 32 * kK2Warps;
constexpr int kChunk = 32;            // samples of an FP32 partial sum
constexpr int kMaxSpan = kLaneCap / 32 / kK2Warps + 2;  // groups a warp's share of a tile touches at most

// What the lanes of a group need of their parents.
template <typename T>
struct ParentRow;
template <>
struct ParentRow<float> {
    float r, lr, alpha_r;
    float r2;  // rounded from FP64
};
template <>
struct ParentRow<double> {
    double r, lr, alpha_r;
};

// The set of a CTA column (SetTable::cta_first), its rank in the set and the
// set's number of CTAs; every thread of the CTA calls it.
__device__ __forceinline__ int find_set(const SetTable* table, int sets, int& rank, int& ctas)
{
    __shared__ int found[3];
    const int x = (int)blockIdx.x;
    for (int s = threadIdx.x; s < sets; s += blockDim.x) {
        const int first = table->cta_first[s], next = table->cta_first[s + 1];
        if (x >= first && x < next) {
            found[0] = s;
            found[1] = x - first;
            found[2] = next - first;
        }
    }
    __syncthreads();
    rank = found[1];
    ctas = found[2];
    return found[0];
}

// Shared memory of a CTA: records, the T-typed log S coefficients, the pre-scaled FP32 rows with
// their edge rows (FP32 build), knots, parents, the warps' sums, Sobol directions.
template <typename T>
__host__ __device__ inline size_t k2_smem_bytes(int n)
{
    auto a16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    return sizeof(K2Rec<T>) * kK2Threads + a16(sizeof(T) * 4 * (size_t)(n - 1)) +
           (sizeof(T) == sizeof(float) ? sizeof(float4) * (size_t)(n + 1) : 0) + a16(sizeof(T) * (size_t)n) +
           sizeof(ParentRow<T>) * kLaneCap + sizeof(double) * 3 * kK2Warps * kMaxSpan * 32 +
           sizeof(uint32_t) * kSetDirsWords;
}

// Grid x: the CTAs of every set side by side, in proportion to their budgets; grid y: parent tiles.
template <typename T, bool SYM, int COUPLING>
__global__ void __launch_bounds__(kK2Threads, (sizeof(T) == 4 ? 3 : 2))
    k2kf_sets_kernel(Phys<T> ph, K2Box<T> box, const double* __restrict__ r_grid, int n,
                     const double* __restrict__ spline, const int32_t* __restrict__ active,
                     const int32_t* __restrict__ count, double* __restrict__ partial,
                     const SetTable* __restrict__ table, int sets)
{
    int rank, ctas;
    const int set = find_set(table, sets, rank, ctas);
    const uint64_t samples = table->samples[set];
    spline += (size_t)set * spline_doubles(n);
    active += (size_t)set * n;
    count += set;
    const int first = (int)blockIdx.y * kLaneCap;
    const int parents = min(kLaneCap, *count - first);
    if (parents <= 0) return;  // the finalize reads the slots below the count only
    const int groups = (parents + 31) >> 5;
    // the CTA's chunks [begin, end) of 32 samples
    const uint64_t chunks = (samples + kChunk - 1) / kChunk;
    const uint64_t begin = chunks * rank / ctas, end = chunks * (rank + 1) / ctas;

    extern __shared__ __align__(16) unsigned char k2_smem[];
    unsigned char* cursor = k2_smem;
    auto carve = [&](size_t bytes) {
        unsigned char* at = cursor;
        cursor += (bytes + 15) & ~(size_t)15;
        return at;
    };
    K2Rec<T>* recs = reinterpret_cast<K2Rec<T>*>(carve(sizeof(K2Rec<T>) * kK2Threads));
    T* cs = reinterpret_cast<T*>(carve(sizeof(T) * 4 * (size_t)(n - 1)));
    float4* rows = sizeof(T) == sizeof(float) ? reinterpret_cast<float4*>(carve(sizeof(float4) * (size_t)(n + 1)))
                                              : nullptr;
    T* xs = reinterpret_cast<T*>(carve(sizeof(T) * (size_t)n));
    ParentRow<T>* prow = reinterpret_cast<ParentRow<T>*>(carve(sizeof(ParentRow<T>) * kLaneCap));
    double* sums = reinterpret_cast<double*>(carve(sizeof(double) * 3 * kK2Warps * kMaxSpan * 32));
    uint32_t* st = reinterpret_cast<uint32_t*>(carve(sizeof(uint32_t) * kSetDirsWords));

    const double h64 = (spline[n - 1] - spline[0]) / (double)(n - 1);
    const double* src_coef = spline + n + 4 * (size_t)(n - 1);  // log S block
    for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = (T)spline[i];
    for (int i = threadIdx.x; i < 4 * (n - 1); i += blockDim.x) cs[i] = (T)src_coef[i];
    if constexpr (sizeof(T) == sizeof(float)) stage_fast_rows(rows, src_coef, n, h64);
    for (int i = threadIdx.x; i < 32 * groups; i += blockDim.x) {
        const double r = i < parents ? r_grid[active[first + i]] : 1.0;
        ParentRow<T> p;
        p.r = (T)r;
        if constexpr (sizeof(T) == sizeof(float)) p.r2 = (T)(r * r);
        p.lr = (T)log(r);
        p.alpha_r = alpha_of_log(p.lr, ph);
        prow[i] = p;
    }
    for (int i = threadIdx.x; i < 3 * kK2Warps * kMaxSpan * 32; i += blockDim.x) sums[i] = 0.0;
    for (int i = threadIdx.x; i < kSetDirsWords; i += blockDim.x)
        st[i] = table->dirs[set][i];
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
    if constexpr (sizeof(T) == sizeof(float)) fs = fast_spline(rows, n, spline[0], h64);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the groups of a warp's shares start at the same one for every tile: floor(floor(w g t / 8) / t)
    // = floor(w g / 8)
    const int group0 = warp * groups / kK2Warps;
    double* my_sums = sums + (size_t)warp * kMaxSpan * 96;
    for (uint64_t c0 = begin; c0 < end; c0 += kK2Warps) {
        const int tile = (int)(end - c0 < kK2Warps ? end - c0 : kK2Warps);  // chunks
        const uint64_t local = c0 * kChunk + threadIdx.x;
        if (warp < tile) {
            if constexpr (sizeof(T) == sizeof(float)) {
                // pair layout: the fields of samples 2p and 2p+1 side by side (a padding sample
                // past the budget carries zero weight)
                float rec[kRecLen];
                k2_prepare<float>(s, box, st, st + 120, local, local < samples, rec);
                float* dst = reinterpret_cast<float*>(recs) + (size_t)(threadIdx.x >> 1) * (2 * kRecLen) +
                             (threadIdx.x & 1);
#pragma unroll
                for (int f = 0; f < kRecLen; ++f) dst[2 * f] = rec[f];
            } else {
                k2_prepare<T>(s, box, st, st + 120, local, local < samples, recs[threadIdx.x].v);
            }
        }
        __syncthreads();
        int u = warp * groups * tile / kK2Warps;
        const int u_end = (warp + 1) * groups * tile / kK2Warps;
        while (u < u_end) {
            const int group = u / tile;
            const int from = u - group * tile;
            const int to = min(tile, from + (u_end - u));
            u += to - from;
            if (32 * group + lane < parents) {
                const ParentRow<T> row = prow[32 * group + lane];
                double a_tot = 0.0, a_kf = 0.0, a_sq = 0.0;
                if constexpr (sizeof(T) == sizeof(float)) {
                    K2ParentF P;
                    P.r = row.r;
                    P.r2 = row.r2;
                    P.lr = row.lr;
                    P.two_r = 2.0f * row.r;
                    P.four_r = 4.0f * row.r;
                    P.alpha_r = row.alpha_r;
                    f2 sq = bc2(0.0f);  // variance estimate only: plain sum per share
                    for (int c = from; c < to; ++c) {
                        const float4* pr = reinterpret_cast<const float4*>(recs) + (size_t)c * (kChunk / 2) * (kRecLen / 2);
                        // FP32x2 partial sums of 16 pairs (32 samples), folded into FP64: the
                        // rounding of a 32-term FP32 sum instead of compensated summation.  The
                        // sums are of K2 + Kf and of Kf (K2 is their difference, formed once at
                        // the end): the total is needed anyway for the variance, and this saves
                        // the finite-test select of K2 per sample
                        f2 ptot = bc2(0.0f), pkf = bc2(0.0f);
                        for (int j = 0; j < kChunk / 2; ++j) {
                            f2 kfw, tot;
                            k2_pair_fast<SYM, COUPLING>(fs, ph, P, pr + (kRecLen / 2) * j, kfw, tot);
                            ptot = add2(ptot, tot);
                            pkf = add2(pkf, kfw);
                            sq = fma2(tot, tot, sq);
                        }
                        a_tot += (double)ptot.x + (double)ptot.y;
                        a_kf += (double)pkf.x + (double)pkf.y;
                    }
                    a_sq = (double)sq.x + (double)sq.y;
                } else {
                    K2Parent<T> P;
                    P.r = row.r;
                    P.r2 = row.r * row.r;
                    P.lr = row.lr;
                    P.two_r = (T)2 * row.r;
                    P.alpha_r = row.alpha_r;
                    for (int c = from; c < to; ++c) {
                        Kahan<T> sk2, skf;
                        sk2.reset();
                        skf.reset();
                        T sq = (T)0;
                        for (int j = 0; j < kChunk; ++j) {
                            T k2w, kfw;
                            k2_point<T, SYM>(s, ph, P, recs[c * kChunk + j].v, k2w, kfw);
                            sk2.add(k2w);
                            skf.add(kfw);
                            const T tot = k2w + kfw;
                            sq += tot * tot;
                        }
                        a_tot += (double)sk2.sum - (double)sk2.comp;
                        a_kf += (double)skf.sum - (double)skf.comp;
                        a_sq += (double)sq;
                    }
                }
                double* o = my_sums + 96 * (group - group0) + lane;
                o[0] += a_tot;
                o[32] += a_kf;
                o[64] += a_sq;
            }
        }
        __syncthreads();
    }
    // the warps' sums of each parent in warp order
    double* out = partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * min(n, kLaneCap) * 3;
    for (int i = threadIdx.x; i < parents; i += blockDim.x) {
        const int group = i >> 5;
        double v[3] = {0.0, 0.0, 0.0};
        for (int w = 0; w < kK2Warps; ++w) {
            const int g0 = w * groups / kK2Warps;
            // the last group of warp w's share of a full tile
            const int g1 = ((w + 1) * groups + kK2Warps - 1) / kK2Warps - 1;
            if (group < g0 || group > g1) continue;
            const double* q = sums + ((size_t)w * kMaxSpan + (group - g0)) * 96 + (i & 31);
            v[0] += q[0];
            v[1] += q[32];
            v[2] += q[64];
        }
        out[3 * i] = sizeof(T) == sizeof(float) ? v[0] - v[1] : v[0];
        out[3 * i + 1] = v[1];
        out[3 * i + 2] = v[2];
    }
}

// One warp per (set blockIdx.y, active parent): lanes add strided partials of the set's CTAs, then a
// fixed shuffle tree combines them (the order does not depend on timing).
__global__ void __launch_bounds__(256) k2kf_finalize_sets_kernel(const double* __restrict__ partial, int blocks, int n,
                                                                 const int32_t* __restrict__ active,
                                                                 const int32_t* __restrict__ count,
                                                                 const SetTable* __restrict__ table,
                                                                 double* __restrict__ out)
{
    const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int set = blockIdx.y;
    if (slot >= n || slot >= count[set]) return;
    const int cap = min(n, kLaneCap), tile = slot / kLaneCap;
    const double* p = partial + ((size_t)tile * blocks * cap + (slot - tile * kLaneCap)) * 3;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int c = table->cta_first[set] + lane; c < table->cta_first[set + 1]; c += 32) {
        const double* q = p + 3 * (size_t)cap * c;
        s0 += q[0];
        s1 += q[1];
        s2 += q[2];
    }
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, o);
        s1 += __shfl_down_sync(0xffffffffu, s1, o);
        s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        double* o = out + 3 * ((size_t)set * n + active[(size_t)set * n + slot]);
        o[0] = s0;
        o[1] = s1;
        o[2] = s2;
    }
}

inline int parent_tiles_of(int points) { return (points + kLaneCap - 1) / kLaneCap; }

}  // namespace

SetsLayout sets_layout(int points, int sets, int waves)
{
    SetsLayout L;
    L.parent_tiles = parent_tiles_of(points);
    L.lanes = points < kLaneCap ? points : kLaneCap;
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (sms < 1) sms = 148;
    // about `waves` waves of the FP32 kernel's three CTAs per SM over all parent tiles
    const long blocks = (long)(waves < 1 ? 1 : waves) * 3 * sms / L.parent_tiles;
    L.blocks = (int)(blocks < sets ? sets : blocks);
    return L;
}

void sets_ctas(const SetsLayout& L, bool fp64, int points, const int64_t* samples, int sets, uint16_t* first)
{
    // the layout is sized for three CTAs per SM; the FP64 build (registers) and long FP32 tables
    // (shared memory) have two, the longest one
    const size_t smem = fp64 ? k2_smem_bytes<double>(points) : k2_smem_bytes<float>(points);
    const int fit = (int)((size_t)(228 << 10) / (smem + 1024));
    const int per_sm = fit < 1 ? 1 : fp64 ? (fit < 2 ? fit : 2) : (fit < 3 ? fit : 3);
    const int blocks = L.blocks / 3 * per_sm;
    int64_t left = blocks > sets ? blocks - sets : 0;
    double total = 0.0;
    for (int s = 0; s < sets; ++s) total += (double)samples[s];
    const int64_t spare = left;
    int at = 0;
    for (int s = 0; s < sets; ++s) {
        first[s] = (uint16_t)at;
        const int64_t chunks = (samples[s] + kChunk - 1) / kChunk;
        int64_t extra = total > 0.0 ? (int64_t)((double)spare * ((double)samples[s] / total)) : 0;
        if (extra > left) extra = left;
        left -= extra;
        at += (int)(1 + extra < chunks ? 1 + extra : (chunks < 1 ? 1 : chunks));
    }
    first[sets] = (uint16_t)at;
}

cudaError_t launch_k2kf_sets(const nlo_bk_params& p, const double* r, int points, int sets, const double* spline,
                             const int32_t* active, const int32_t* counts, const nlo_bk_box& box, int blocks,
                             const SetTable* table, double* out, double* partial, cudaStream_t stream, bool cleared)
{
    cudaError_t e = cleared ? cudaSuccess : cudaMemsetAsync(out, 0, sizeof(double) * 3 * (size_t)points * sets, stream);
    if (e != cudaSuccess) return e;
    const int tiles = parent_tiles_of(points);
    e = dispatch_variant(p, [&](auto t, auto sym, auto c) {
        using T = decltype(t);
        constexpr bool SYM = decltype(sym)::value;
        constexpr int COUPLING = decltype(c)::value;
        const void* fn = (const void*)k2kf_sets_kernel<T, SYM, COUPLING>;
        const size_t smem = k2_smem_bytes<T>(points);
        cudaError_t err = raise_dynamic_smem(fn, smem);
        if (err == cudaSuccess) err = prefer_shared_carveout(fn);
        if (err != cudaSuccess) return err;
        k2kf_sets_kernel<T, SYM, COUPLING><<<dim3((unsigned)blocks, (unsigned)tiles), kK2Threads, smem, stream>>>(
            make_phys<T>(p), make_box<T>(p, box, SYM), r, points, spline, active, counts, partial, table, sets);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    k2kf_finalize_sets_kernel<<<dim3((points * 32 + 255) / 256, sets), 256, 0, stream>>>(partial, blocks, points,
                                                                                         active, counts, table, out);
    return cudaGetLastError();
}

}  // namespace nlo
