// Log-log natural cubic splines of the evolving amplitude (FP64), the active
// parent list, and the device Sobol draw.
//
// Spline: restates numerics/interpolation.py:10-121 (natural cubic spline with a
// Thomas solve, log-log table with -40 for non-positive values) for the two
// evolution rows of bk/evolution.py:548-560: log N with N clamped to [0,1], and
// log S with S = 1 - N clamped to [0,1], evaluated as log1p(-N) so that S close to
// 1 keeps the relative precision of N.  One CTA per row pair; the two rows' Thomas
// sweeps run concurrently in two warps, as scans over the warp.

#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"
#include "sobol.cuh"

namespace nlo {

// s_i = c_i + a_i s_{i-1} over i = 0..m-1 (REVERSE: s_i = c_i + a_i s_{i+1} from the other end), in
// place over c, by one warp: a lane composes the affine maps of its consecutive elements, a
// warp scan composes the lanes', and each lane walks its elements again from its carry-in.
// m = 398: 13 elements twice and 5 scan steps instead of a chain of 398.
template <bool REVERSE>
__device__ __forceinline__ void warp_affine_scan(const double* a, double* c, int m)
{
    const int lane = threadIdx.x & 31;
    const int per = (m + 31) / 32;
    const int begin = min(lane * per, m), end = min(begin + per, m);
    auto at = [&](int i) { return REVERSE ? m - 1 - i : i; };
    double A = 1.0, C = 0.0;
    for (int i = begin; i < end; ++i) {
        const int k = at(i);
        C = fma(a[k], C, c[k]);
        A *= a[k];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double A1 = __shfl_up_sync(0xffffffffu, A, o), C1 = __shfl_up_sync(0xffffffffu, C, o);
        if (lane >= o) {
            C = fma(A, C1, C);
            A *= A1;
        }
    }
    double carry = __shfl_up_sync(0xffffffffu, C, 1);
    if (lane == 0) carry = 0.0;
    for (int i = begin; i < end; ++i) {
        const int k = at(i);
        carry = fma(a[k], carry, c[k]);
        c[k] = carry;
    }
}

// factor: [2][n] = 1/denominator and upper coefficient of the Thomas sweep for
// the natural-spline system on the knots log r (it depends on the grid only).
// With compute_factor set, one warp forms it first (and stores it for later calls).
// One CTA per set (blockIdx.x): row N.at(set), tables at out + set * spline_doubles(n), its own
// factorisation copy at factor + set * 2n.  k1 and k2kf (optional): the sums of the right-hand side
// that begins with this refit, cleared here instead of by two memsets on its critical path.
// What bounds it: the latency of the dependent sweeps (33 us for 400 knots with one thread per
// row; the scans leave about 8).
__global__ void __launch_bounds__(256) splines_kernel(const double* __restrict__ r, RowsArg rows,
                                                      int n, int force_positive, double* __restrict__ factor,
                                                      int compute_factor, double* __restrict__ out,
                                                      double* __restrict__ k1, double* __restrict__ k2kf)
{
    const double* __restrict__ N = rows.at(blockIdx.x);
    factor += (size_t)blockIdx.x * 2 * n;
    out += (size_t)blockIdx.x * spline_doubles(n);
    extern __shared__ double smem[];
    double* x = smem;             // [n]
    double* y = x + n;            // [2][n]
    double* sol = y + 2 * n;      // [2][n]
    double* low = sol + 2 * n;    // [n]
    double* up = low + n;         // [n]
    const int m = n - 2;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        x[i] = log(r[i]);
        out[i] = x[i];
        const double v = N[i];
        // log N row: N > 1 -> 1; force_positive: N < 0 -> 0
        double vn = v > 1.0 ? 1.0 : v;
        if (force_positive && vn < 0.0) vn = 0.0;
        y[i] = vn > 0.0 ? log(vn) : kMinLog;
        // log S row: S = 1 - N; S < 0 -> 0; force_positive: S > 1 -> 1
        double ns = v;
        if (force_positive && ns < 0.0) ns = 0.0;
        y[n + i] = ns < 1.0 ? log1p(-ns) : kMinLog;
        if (k1) k1[(size_t)blockIdx.x * n + i] = 0.0;
    }
    if (k2kf)
        for (int i = threadIdx.x; i < 3 * n; i += blockDim.x) k2kf[(size_t)blockIdx.x * 3 * n + i] = 0.0;
    __syncthreads();
    if (compute_factor && threadIdx.x < 32 && m >= 1) {
        // denominators of the forward sweep (interpolation.py:124-149): lane l its own stretch,
        // entered kFactorWarmup elements earlier from the undivided denominator.  The recurrence
        // forgets its start (a factor of 0.07 a step on the uniform grid, under 0.45 on any), so
        // the stretch is the serial sweep's to the last digits.
        constexpr int kFactorWarmup = 48;
        const int per = (m + 31) / 32;
        const int begin = min((int)threadIdx.x * per, m), end = min(begin + per, m);
        int i = max(0, begin - kFactorWarmup);
        double inv = 1.0 / (2.0 * ((x[i + 1] - x[i]) + (x[i + 2] - x[i + 1])));
        if (i == begin && begin < end) factor[i] = inv;
        for (++i; i < end; ++i) {
            const double h = x[i + 1] - x[i];
            const double upper_prev = h * inv;
            if (i > begin || begin == 0) factor[n + i - 1] = upper_prev;
            inv = 1.0 / (2.0 * (h + (x[i + 2] - x[i + 1])) - h * upper_prev);
            if (i >= begin) factor[i] = inv;
        }
        if (begin < end && end < m) factor[n + end - 1] = (x[end + 1] - x[end]) * inv;
    }
    __syncthreads();
    // The forward sweep s_i = (b_i - h_i s_{i-1}) / d_i as s_i = c_i + a_i s_{i-1} with
    // c_i = b_i / d_i and a_i = -h_i / d_i; the back substitution likewise with the negated
    // upper diagonal.
    for (int item = threadIdx.x; item < 2 * m; item += blockDim.x) {
        const int row = item / m, i = item - row * m;
        const double* yy = y + row * n;
        sol[row * n + i] =
            6.0 * ((yy[i + 2] - yy[i + 1]) / (x[i + 2] - x[i + 1]) - (yy[i + 1] - yy[i]) / (x[i + 1] - x[i])) * factor[i];
        if (row == 0) {
            low[i] = i > 0 ? -(x[i + 1] - x[i]) * factor[i] : 0.0;
            up[i] = i < m - 1 ? -factor[n + i] : 0.0;
        }
    }
    __syncthreads();
    // warp 0 solves row 0, warp 1 row 1
    if (threadIdx.x < 64 && m >= 1) {
        double* s = sol + (threadIdx.x >> 5) * n;
        warp_affine_scan<false>(low, s, m);
        __syncwarp();
        warp_affine_scan<true>(up, s, m);
    }
    __syncthreads();
    for (int item = threadIdx.x; item < 2 * (n - 1); item += blockDim.x) {
        const int row = item / (n - 1);
        const int i = item - row * (n - 1);
        const double* yy = y + row * n;
        const double* s = sol + row * n;
        const double h = x[i + 1] - x[i];
        const double sl = i == 0 ? 0.0 : s[i - 1];
        const double sr = i == n - 2 ? 0.0 : s[i];
        double* c = out + n + (size_t)row * 4 * (n - 1) + 4 * (size_t)i;
        c[0] = yy[i];
        c[1] = (yy[i + 1] - yy[i]) / h - h * (2.0 * sl + sr) / 6.0;
        c[2] = sl / 2.0;
        c[3] = (sr - sl) / (6.0 * h);
    }
}

// The active parents of each row (index > 0 and N <= 0.99999, bk/evolution.py:501; index % shards ==
// shard), compacted in index order by a ballot scan; one CTA per set (blockIdx.x).
__global__ void __launch_bounds__(1024) active_kernel(RowsArg rows, int n, int shard, int shards,
                                                      int32_t* __restrict__ active, int32_t* __restrict__ count)
{
    const double* __restrict__ N = rows.at(blockIdx.x);
    active += (size_t)blockIdx.x * n;
    count += blockIdx.x;
    __shared__ int warp_counts[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int start = 0; start < n; start += blockDim.x) {
        const int i = start + threadIdx.x;
        const bool on = i < n && i > 0 && N[i] <= 0.99999 && i % shards == shard;
        const unsigned mask = __ballot_sync(0xffffffffu, on);
        if (lane == 0) warp_counts[warp] = __popc(mask);
        __syncthreads();
        int offset = base;
        for (int w = 0; w < warp; ++w) offset += warp_counts[w];
        if (on) active[offset + __popc(mask & ((1u << lane) - 1u))] = i;
        __syncthreads();
        if (threadIdx.x == 0) {
            int total = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) total += warp_counts[w];
            base += total;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = base;
}

template <typename T>
__global__ void sobol_draw_kernel(SobolDirsArg dirs, uint64_t offset, uint64_t n, T* __restrict__ out)
{
    const int d = dirs.dims;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t index = offset + k;
        for (int j = 0; j < d; ++j) {
            const uint32_t bits = sobol_bits(dirs.state[j], dirs.shift[j], index);
            out[k * d + j] = sobol_unit<T>(bits, index);
        }
    }
}

cudaError_t launch_splines(const double* r, const RowsArg& N, int n, int sets, int force_positive, double* factor,
                           int compute_factor, double* out, cudaStream_t stream, double* k1, double* k2kf)
{
    const size_t smem = sizeof(double) * 7 * (size_t)n;
    const cudaError_t e = raise_dynamic_smem((const void*)splines_kernel, smem);
    if (e != cudaSuccess) return e;
    splines_kernel<<<sets, 256, smem, stream>>>(r, N, n, force_positive, factor, compute_factor, out, k1, k2kf);
    return cudaGetLastError();
}

cudaError_t launch_active(const RowsArg& N, int n, int sets, int shard, int shards, int32_t* active, int32_t* count,
                          cudaStream_t stream)
{
    active_kernel<<<sets, 1024, 0, stream>>>(N, n, shard, shards, active, count);
    return cudaGetLastError();
}

cudaError_t launch_sobol(const SobolDirsArg& dirs, uint64_t offset, uint64_t n, int precision, void* out,
                         cudaStream_t stream)
{
    const int threads = 256;
    uint64_t blocks64 = (n + threads - 1) / threads;
    const int blocks = (int)(blocks64 > 65535 ? 65535 : (blocks64 == 0 ? 1 : blocks64));
    if (precision == NLO_PRECISION_FP64)
        sobol_draw_kernel<double><<<blocks, threads, 0, stream>>>(dirs, offset, n, (double*)out);
    else
        sobol_draw_kernel<float><<<blocks, threads, 0, stream>>>(dirs, offset, n, (float*)out);
    return cudaGetLastError();
}

}  // namespace nlo
