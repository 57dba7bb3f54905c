// NLO DIS kernels (sm_100a): BK-table preparation, pointwise integrands, the tensor
// Gauss-Legendre rule of the 2D terms, and the device Vegas iteration.
//
// Vegas (numerics/integration.py:120-589, 804-866) runs entirely on the device: one
// iteration kernel per round maps scrambled Sobol points through the current grid,
// evaluates the integrand, and leaves per-CTA partial sums of w, w^2 and the |w| / count
// histograms; one finalize CTA per integral reduces the partials in a fixed order,
// re-bins the grid and updates the inverse-variance-weighted estimate and the
// convergence flag.  A converged integral makes the remaining rounds no-ops, so the host
// enqueues all rounds without synchronising.  Many integrals (jobs) of one term run in
// the same launches (grid.y = job).  Every reduction has a fixed order, so results are
// bit-reproducible run to run.
#include <cuda_runtime.h>

#include "dis_internal.h"
#include "dis_terms.cuh"
#include "sobol.cuh"
#include "vegas_common.cuh"
#include "vegas_sampling.cuh"

namespace nlo {
namespace dis {

// ===========================================================================
// Table preparation (dipole/amplitude.py:48-83, 215-252)

__global__ void table_prepare_kernel(const double* __restrict__ r, const double* __restrict__ y,
                                     const double* __restrict__ N, int nr, int ny, double y0, int interp,
                                     double* table)
{
    const TableView v = table_view(table, nr, ny);
    double* hdr = table;
    double* tr = table + kTableHeader;
    double* tY = tr + nr;
    double* tN = tY + ny;
    double* win = tN + (size_t)ny * nr;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    for (int i = tid; i < nr; i += stride) tr[i] = r[i];
    for (int i = tid; i < ny; i += stride) tY[i] = y[i] + y0;
    for (size_t i = tid; i < (size_t)ny * nr; i += stride) tN[i] = N[i];
    if (tid == 0) {
        for (int k = 0; k < kTableHeader; ++k) hdr[k] = 0.0;
        hdr[kHdrNr] = nr;
        hdr[kHdrNy] = ny;
        hdr[kHdrInitialized] = 0.0;
        hdr[kHdrInitY] = -1.0;
        hdr[kHdrMaxrInterp] = -1.0;
        hdr[kHdrRmin] = r[0];
        hdr[kHdrRmax] = r[nr - 1];
        hdr[kHdrYmin] = y[0] + y0;
        hdr[kHdrYmax] = y[ny - 1] + y0;
        hdr[kHdrLogR0] = ::log(r[0]);
        hdr[kHdrInvDlogR] = (nr - 1) / (::log(r[nr - 1]) - ::log(r[0]));
        hdr[kHdrInterp] = interp;
        hdr[kHdrY0] = y[0] + y0;
        hdr[kHdrInvDY] = ny > 1 ? (ny - 1) / ((y[ny - 1] + y0) - (y[0] + y0)) : 0.0;
    }
    // window weights: second derivatives of the natural spline through the 7/9 window
    // points as linear maps of the window values (one Thomas solve per unit vector)
    for (int i = tid; i < nr - 1; i += stride) {
        const bool upper = i + 3 > nr - 1;
        const int points = upper ? 9 : 7;
        int start = upper ? nr - 9 : i - 3;
        start = start < 0 ? 0 : start;
        const int j = i - start;
        double h[kWindowMax - 1];
        for (int k = 0; k < points - 1; ++k) h[k] = r[start + k + 1] - r[start + k];
        double* w = win + (size_t)i * kWindowStride;
        w[0] = start;
        w[1] = points;
        for (int k = 0; k < 2 * kWindowMax; ++k) w[2 + k] = 0.0;
        const int m = points - 2;  // interior unknowns
        for (int unit = 0; unit < points; ++unit) {
            double c[kWindowMax], d[kWindowMax];
            for (int q = 0; q < m; ++q) {
                // rhs_q = 6 ((e_{q+2} - e_{q+1})/h_{q+1} - (e_{q+1} - e_q)/h_q)
                const double e0 = unit == q ? 1.0 : 0.0;
                const double e1 = unit == q + 1 ? 1.0 : 0.0;
                const double e2 = unit == q + 2 ? 1.0 : 0.0;
                const double rhs = 6.0 * ((e2 - e1) / h[q + 1] - (e1 - e0) / h[q]);
                const double diag = 2.0 * (h[q] + h[q + 1]);
                if (q == 0) {
                    c[q] = m > 1 ? h[1] / diag : 0.0;
                    d[q] = rhs / diag;
                } else {
                    const double den = diag - h[q] * c[q - 1];
                    c[q] = q < m - 1 ? h[q + 1] / den : 0.0;
                    d[q] = (rhs - h[q] * d[q - 1]) / den;
                }
            }
            double M[kWindowMax];
            M[0] = 0.0;
            M[points - 1] = 0.0;
            double next = d[m - 1];
            M[m] = next;
            for (int q = m - 2; q >= 0; --q) {
                next = d[q] - c[q] * next;
                M[q + 1] = next;
            }
            w[2 + unit] = M[j];
            w[2 + kWindowMax + unit] = M[j + 1];
        }
    }
    (void)v;
}

// Per-row coefficients of the local splines: for table row k and r interval i, the
// window spline through row k's values (second derivatives from the window weights),
// in the power form a + b dx + c dx^2 + d dx^3 on [r_i, r_{i+1}).
__global__ void table_local_kernel(double* table, int nr, int ny)
{
    const TableView v = table_view(table, nr, ny);
    double* local = table + (v.local - table);
    const int64_t total = (int64_t)ny * (nr - 1);
    for (int64_t item = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; item < total;
         item += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(item / (nr - 1));
        const int i = (int)(item - (int64_t)k * (nr - 1));
        const double* w = v.window + (size_t)i * kWindowStride;
        const int start = (int)w[0];
        const int points = (int)w[1];
        const int j = i - start;
        const double* vals = v.N + (size_t)k * nr + start;
        double mj = 0.0, mj1 = 0.0;
        for (int q = 0; q < points; ++q) {
            mj = fma(w[2 + q], vals[q], mj);
            mj1 = fma(w[2 + kWindowMax + q], vals[q], mj1);
        }
        const double vj = vals[j], vj1 = vals[j + 1];
        const double h = v.r[i + 1] - v.r[i];
        double* out = local + (size_t)item * 4;
        out[0] = vj;
        out[1] = (vj1 - vj) / h - h * (2.0 * mj + mj1) / 6.0;
        out[2] = mj / 2.0;
        out[3] = (mj1 - mj) / (6.0 * h);
    }
}

// initialize_interpolation (dipole/amplitude.py:105-133) and _find_maxr_interpolate
// (:254-272): one CTA.  Threads evaluate the local amplitude at the knots (the end knots
// nudged inwards by 1e-4), form the spline's right-hand sides and coefficients and stage the
// knots in shared memory; one thread runs the two tridiagonal recurrences.  The search's next
// radii depend on the amplitudes only at the at most 14 reductions of its step, so a warp
// evaluates the 32 radii that follow if there is none and goes on from the first reduction.
// What bounds it: latency of the recurrences' divisions.  One thread doing all of it took 293 us
// at 400 knots and 72 us at 64; this takes 103 and 35 us, with every value's operations and their
// order unchanged (amplitudes and the radius found are the same to the last bit).
__global__ void table_initialize_kernel(double* table, int nr, int ny, double Y)
{
    extern __shared__ double smem[];
    double* vals = smem;        // [nr]
    double* cc = smem + nr;     // [nr]
    double* dd = smem + 2 * nr; // [nr]
    TableView v = table_view(table, nr, ny);
    double* hdr = table;
    if (threadIdx.x == 0) {
        hdr[kHdrInitialized] = 0.0;
        hdr[kHdrInitY] = -1.0;
        hdr[kHdrMaxrInterp] = -1.0;
    }
    __syncthreads();
    double Yv = Y;
    if (Yv >= 0.0 && Yv <= hdr[kHdrYmin]) Yv = hdr[kHdrYmin];
    for (int k = threadIdx.x; k < nr; k += blockDim.x) {
        double rr = v.r[k];
        if (k == 0) rr *= 1.0001;
        if (k == nr - 1) rr *= 0.9999;
        vals[k] = table_amplitude(v, rr, Yv);
    }
    __syncthreads();
    // natural spline through (r_k, vals_k): right-hand sides, and the coefficients' parts without
    // second derivatives
    double* g = table + (v.global - table);
    const int m = nr - 2;
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
        const double h0 = v.r[q + 1] - v.r[q], h1 = v.r[q + 2] - v.r[q + 1];
        dd[q] = 6.0 * ((vals[q + 2] - vals[q + 1]) / h1 - (vals[q + 1] - vals[q]) / h0);
    }
    for (int k = threadIdx.x; k < nr - 1; k += blockDim.x) {
        g[4 * k + 0] = vals[k];
        g[4 * k + 1] = (vals[k + 1] - vals[k]) / (v.r[k + 1] - v.r[k]);
    }
    __syncthreads();
    double* rs = vals;  // the knots from here on
    for (int k = threadIdx.x; k < nr; k += blockDim.x) rs[k] = v.r[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        // interior second derivatives by Thomas, back substitution into dd (dd[q] = M_{q+1})
        double c = 0.0, d = 0.0;
        for (int q = 0; q < m; ++q) {
            const double h0 = rs[q + 1] - rs[q], h1 = rs[q + 2] - rs[q + 1];
            const double diag = 2.0 * (h0 + h1);
            const double den = q == 0 ? diag : diag - h0 * c;
            d = (q == 0 ? dd[q] : dd[q] - h0 * d) / den;
            c = q < m - 1 ? h1 / den : 0.0;
            cc[q] = c;
            dd[q] = d;
        }
        for (int q = m - 2; q >= 0; --q) {
            d = dd[q] - cc[q] * d;
            dd[q] = d;
        }
        hdr[kHdrInitY] = Yv;
        hdr[kHdrInitialized] = 1.0;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nr - 1; k += blockDim.x) {
        const double mk = k == 0 ? 0.0 : dd[k - 1];
        const double mk1 = k + 1 == nr - 1 ? 0.0 : dd[k];
        const double h = rs[k + 1] - rs[k];
        g[4 * k + 1] = g[4 * k + 1] - h * (2.0 * mk + mk1) / 6.0;
        g[4 * k + 2] = mk / 2.0;
        g[4 * k + 3] = (mk1 - mk) / (6.0 * h);
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    constexpr int kSteps = 41;
    const int lane = threadIdx.x;
    v.r = rs;
    const TableRow row = table_row(v, Yv);
    const double rmax = hdr[kHdrRmax];
    double step = 2.0, previous = 0.1, rr = 0.01;
    double found = -1.0;
    int it = 0;
    while (it < kSteps) {  // at least one step a pass
        double mine = rr;
        for (int j = 0; j < lane; ++j) mine += step;
        const bool stop = it + lane >= kSteps || mine > rmax;
        const bool event = stop || table_amplitude_at(v, row, mine) >= 0.99999;
        const unsigned events = __ballot_sync(0xffffffffu, event);
        if (events == 0) {
            previous = __shfl_sync(0xffffffffu, mine, 31);
            rr = previous + step;
            it += 32;
            continue;
        }
        const int first = __ffs(events) - 1;
        const double at = __shfl_sync(0xffffffffu, mine, first);
        const double before = __shfl_sync(0xffffffffu, mine, first > 0 ? first - 1 : 0);
        if (__shfl_sync(0xffffffffu, (int)stop, first)) break;
        if (step < 1e-2) {
            found = at;
            break;
        }
        step /= 1.5;
        if (first > 0) previous = before;
        rr = previous + step;
        it += first + 1;
    }
    if (lane == 0) hdr[kHdrMaxrInterp] = found;
}

// ===========================================================================
// Pointwise integrands (the reference's dis_*_integrand operators)

constexpr int kPointsThreads = 128;

// A warp takes per_warp points at a time (32 but for the nested FP32 terms, see launch_points_t).
// Eight CTAs per SM (64 registers) in FP32, four in FP64: the terms are latency-bound.  200,000 points
// of I1, I2 and I3: 11.9, 14.4 and 17.8 us in FP32, 27.3, 42.0 and 59.0 in FP64; bounded for one CTA
// (130 to 230 registers) 17.5, 20.6, 23.7 and 42.9, 58.2, 80.0, and FP64 at eight loses 2 us to spills
// on few points.
template <typename T, int TERM>
__global__ void __launch_bounds__(kPointsThreads, (sizeof(T) == 4 ? 8 : 4))
    points_kernel(const DisArgs<T> args, InnerRule rule, const double* __restrict__ x, int64_t n, int per_warp,
                  double* __restrict__ out)
{
    constexpr int D = term_dims(TERM);
    __shared__ __align__(16) unsigned char raw[sizeof(DisArgs<T>)];
    DisArgs<T>& a = *reinterpret_cast<DisArgs<T>*>(raw);
    __shared__ WarpShared<T, TERM, kPointsThreads> ws;
    if (threadIdx.x == 0) a = args;
    ws.stage(rule);
    __syncthreads();
    // whole warps stay in the loop: a nested FP32 term is evaluated by its warp
    const int lane = threadIdx.x & 31, warps = kPointsThreads / 32;
    const int64_t stride = (int64_t)gridDim.x * warps * per_warp;
    for (int64_t base = (blockIdx.x * (int64_t)warps + (threadIdx.x >> 5)) * per_warp; base < n; base += stride) {
        const int64_t i = base + lane;
        const bool on = lane < per_warp && i < n;
        double xl[D];
#pragma unroll
        for (int d = 0; d < D; ++d) xl[d] = on ? x[i * D + d] : 0.5;
        const double v = (double)term_value_warp<T, TERM>(a, on, xl, rule, ws);
        if (on) out[i] = v;
    }
}

template <typename T>
__global__ void amplitude_kernel(const DisArgs<T> a, const double* __restrict__ r, const double* __restrict__ Y,
                                 int64_t n, double* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)amplitude(a, r[i], Y[i]);
}

// ===========================================================================
// Tensor Gauss-Legendre on the unit square, fine and half-order rules
// (custom_kernels/quadrature.py:14-58): one CTA per job, fixed-order reduction.

template <typename T, int TERM>
__global__ void gauss_legendre_kernel(const DisArgs<T>* __restrict__ args, InnerRule rule, GLRules gl,
                                      double* __restrict__ out)
{
    static_assert(term_dims(TERM) == 2, "tensor rule is used for the 2D terms");
    __shared__ __align__(16) unsigned char raw[sizeof(DisArgs<T>)];
    DisArgs<T>& a = *reinterpret_cast<DisArgs<T>*>(raw);
    if (threadIdx.x == 0) a = args[blockIdx.x];
    __shared__ double red[2][32];
    __syncthreads();
    double acc[2] = {0.0, 0.0};
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        const int n = which == 0 ? gl.n_fine : gl.n_coarse;
        const double* xs = which == 0 ? gl.x_fine : gl.x_coarse;
        const double* ws = which == 0 ? gl.w_fine : gl.w_coarse;
        for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
            const int i0 = k / n, i1 = k % n;
            const double xl[2] = {xs[i0], xs[i1]};
            acc[which] += ws[i0] * ws[i1] * (double)term_value<T, TERM>(a, xl, rule);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        double v = acc[which];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[which][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double f = 0.0, c = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            f += red[0][w];
            c += red[1][w];
        }
        out[2 * blockIdx.x + 0] = f;
        out[2 * blockIdx.x + 1] = ::fabs(f - c);
    }
}

// ===========================================================================
// Vegas

// partial layout per (job, block): [total, total2, hist[D][bins]] doubles and
// count[D][bins] int32 in a parallel array
// CTAs per SM the register bound aims at: the FP32 LO and dipole terms are latency-bound and run
// faster at four (64 registers), and so do the nested qqbar-g terms with their nodes on the lanes
// (sigma_r of 24 points 24.8 ms, 25.1 at three); the other qqbar-g terms keep three (80
// registers), where I1 gains nothing from a fourth CTA but spills.
template <typename T, int TERM>
constexpr int vegas_min_blocks()
{
    return sizeof(T) == 4 && (TERM <= kTermDip2 || warp_term<T, TERM>()) ? 4 : 3;
}

template <typename T, int TERM>
__global__ void __launch_bounds__(kVegasThreads, (vegas_min_blocks<T, TERM>())) vegas_iteration_kernel(
    const DisArgs<T>* __restrict__ args, const SobolDirsArg* __restrict__ dirs, InnerRule rule,
    double* __restrict__ state, int state_stride, int bins, uint64_t offset, uint64_t samples, int blocks_per_job,
    double* __restrict__ partial, int32_t* __restrict__ counts)
{
    constexpr int D = term_dims(TERM);
    const int job = blockIdx.y;
    const double* st = state + (size_t)job * state_stride;
    if (st[D * (bins + 1) + kStConverged] != 0.0) return;  // uniform per job

    extern __shared__ __align__(16) unsigned char vsmem[];
    double2* cells = reinterpret_cast<double2*>(vsmem);                  // [D][bins] left end and width
    double* whist = reinterpret_cast<double*>(cells + D * bins);         // [warps][D*bins]
    int32_t* cnt = reinterpret_cast<int32_t*>(whist + (kVegasThreads / 32) * D * bins);  // [D*bins]
    __shared__ double red[2][kVegasThreads / 32];
    __shared__ vegas::SobolWarp<D> sobol;

    const int warps = kVegasThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double fb = (double)bins;
    for (int k = threadIdx.x; k < D * bins; k += blockDim.x) {
        const int e = k + k / bins;
        const double left = st[e], width = st[e + 1] - left;
        cells[k] = make_double2(left, width);
        cnt[k] = 0;
    }
    for (int k = threadIdx.x; k < warps * D * bins; k += blockDim.x) whist[k] = 0.0;
    const SobolDirsArg& sd = dirs[job];
    vegas::stage_sobol(sobol, sd.state, sd.shift, bins);
    __shared__ __align__(16) unsigned char raw[sizeof(DisArgs<T>)];
    DisArgs<T>& a = *reinterpret_cast<DisArgs<T>*>(raw);
    __shared__ WarpShared<T, TERM, kVegasThreads> ws;
    if (threadIdx.x == 0) a = args[job];
    ws.stage(rule);
    __syncthreads();

    // this CTA's share of the round's Sobol indices [first, last), in blocks of 32 aligned indices
    const uint64_t first = offset, last = offset + samples;
    const uint64_t block0 = first >> 5, blocks = ((last + 31) >> 5) - block0;
    const uint64_t share = (blocks + blocks_per_job - 1) / blocks_per_job;
    const uint64_t begin = (uint64_t)blockIdx.x * share;
    const uint64_t end = begin + share < blocks ? begin + share : blocks;
    double tot = 0.0, tot2 = 0.0;
    int whole = 0;
    double* myhist = whist + warp * D * bins;
    for (uint64_t k = begin + warp; k < end; k += warps) {
        const uint32_t base = (uint32_t)((block0 + k) << 5);
        const uint64_t index = (uint64_t)base + lane;
        const bool active = index >= first && index < last;
        double xl[D];
        int bin[D];
        uint32_t bits[D];
        double inv_density = 1.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            bits[d] = vegas::sobol_block_bits(sobol, d, base);
            double rest;
            bin[d] = vegas::grid_position(bits[d], bins, rest);
            const double2 cell = cells[d * bins + bin[d]];
            xl[d] = cell.x + cell.y * (rest * 9.313225746154785e-10);
            inv_density *= fb * cell.y;
        }
        const double w = (double)term_value_warp<T, TERM>(a, active, xl, rule, ws) * inv_density;
        tot += w;
        tot2 += w * w;
        const double aw = ::fabs(w);
        vegas::warp_hist_add(sobol, base, bits, active, bin, bins, aw, myhist, cnt, whole);
    }
    vegas::add_whole_blocks<D>(whole, cnt);
    // block reduction of the sums in warp order
    for (int o = 16; o > 0; o >>= 1) {
        tot += __shfl_down_sync(0xffffffffu, tot, o);
        tot2 += __shfl_down_sync(0xffffffffu, tot2, o);
    }
    if (lane == 0) {
        red[0][warp] = tot;
        red[1][warp] = tot2;
    }
    __syncthreads();
    const size_t pstride = 2 + (size_t)D * bins;
    double* out = partial + ((size_t)job * blocks_per_job + blockIdx.x) * pstride;
    int32_t* cout = counts + (size_t)job * D * bins;  // per-job bin counts, integer atomics
    if (threadIdx.x == 0) {
        double s = 0.0, s2 = 0.0;
        for (int w = 0; w < warps; ++w) {
            s += red[0][w];
            s2 += red[1][w];
        }
        out[0] = s;
        out[1] = s2;
    }
    for (int k = threadIdx.x; k < D * bins; k += blockDim.x) {
        double h = 0.0;
        for (int w = 0; w < warps; ++w) h += whist[w * D * bins + k];
        out[2 + k] = h;
        if (cnt[k]) atomicAdd(&cout[k], cnt[k]);
    }
}

// Sum the per-CTA partials of every job in a fixed order: grid (key chunks, jobs), one
// thread per key (the |w| histogram bins, then total and total^2), looping over the CTAs.
// Per job: sum the per-CTA partials [blocks][keys] over the CTAs.  Each thread takes one
// key and every kReduceSlices-th CTA row (four chains), and the slices of a key are added
// in slice order through shared memory, so the order is fixed; a warp reads 32 consecutive
// keys of a row.
constexpr int kReduceKeys = 32;
constexpr int kReduceSlices = 8;

__global__ void __launch_bounds__(kReduceKeys * kReduceSlices)
    vegas_reduce_kernel(const double* __restrict__ partial, int keys, int blocks_per_job, double* __restrict__ reduced)
{
    __shared__ double sums[kReduceSlices][kReduceKeys];
    const int job = blockIdx.y;
    const int kl = threadIdx.x % kReduceKeys, slice = threadIdx.x / kReduceKeys;
    const int k = blockIdx.x * kReduceKeys + kl;  // 0..keys-1 over [total, total2, hist...]
    double total = 0.0;
    if (k < keys) {
        const double* p = partial + (size_t)job * blocks_per_job * keys + k;
        constexpr int S = kReduceSlices;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int b = slice;
        for (; b + 3 * S < blocks_per_job; b += 4 * S) {
            a0 += p[(size_t)b * keys];
            a1 += p[(size_t)(b + S) * keys];
            a2 += p[(size_t)(b + 2 * S) * keys];
            a3 += p[(size_t)(b + 3 * S) * keys];
        }
        for (; b < blocks_per_job; b += S) a0 += p[(size_t)b * keys];
        total = (a0 + a1) + (a2 + a3);
    }
    sums[slice][kl] = total;
    __syncthreads();
    if (slice == 0 && k < keys) {
        double v = sums[0][kl];
        for (int q = 1; q < kReduceSlices; ++q) v += sums[q][kl];
        reduced[(size_t)job * keys + k] = v;
    }
}

// One CTA per job: adapt the grid (numerics/integration.py:804-866) from the reduced
// histogram and counts, update the combined estimate (:510-582), clear the counts.
__global__ void vegas_finalize_kernel(double* __restrict__ state, int state_stride, int D, int bins,
                                      uint64_t samples, const double* __restrict__ reduced,
                                      int32_t* __restrict__ counts, int warmup, int min_iterations,
                                      double epsrel, double epsabs)
{
    extern __shared__ double fsm[];
    double* smooth = fsm;               // [D*bins]
    double* cum = smooth + D * bins;    // [D*(bins+1)]
    double* ne = cum + D * (bins + 1);  // [D*(bins+1)]
    // the scalar slots in shared memory: one trip to L2 instead of one per dependent access
    __shared__ double sc[kStSlots];
    const int job = blockIdx.x;
    double* st = state + (size_t)job * state_stride;
    double* slots = st + D * (bins + 1);
    int32_t* c = counts + (size_t)job * D * bins;
    if (threadIdx.x < kStSlots) sc[threadIdx.x] = slots[threadIdx.x];
    __syncthreads();
    // combine sets the flag of this very round: every thread has read it before
    const bool converged = sc[kStConverged] != 0.0;
    __syncthreads();
    if (converged) return;
    const int keys = 2 + D * bins;
    const double* red = reduced + (size_t)job * keys;
    // the last thread's chain of divisions runs beside the re-binning
    if (threadIdx.x == blockDim.x - 1) {
        sc[kStEvals] += (double)samples;
        if (!warmup) vegas::combine(sc, red[0], red[1], (double)samples, min_iterations, epsrel, epsabs);
    }
    vegas::rebin(st, red + 2, c, D, bins, smooth, cum, ne);
    __syncthreads();
    for (int k = threadIdx.x; k < D * bins; k += blockDim.x) c[k] = 0;
    __syncthreads();
    if (threadIdx.x < kStSlots) slots[threadIdx.x] = sc[threadIdx.x];
}

__global__ void vegas_init_kernel(double* state, int state_stride, int D, int bins, int jobs, int keep_edges,
                                  int32_t* counts)
{
    const int job = blockIdx.x;
    if (job >= jobs) return;
    for (int k = threadIdx.x; k < D * bins; k += blockDim.x) counts[(size_t)job * D * bins + k] = 0;
    double* st = state + (size_t)job * state_stride;
    if (!keep_edges)
        for (int k = threadIdx.x; k < D * (bins + 1); k += blockDim.x) {
            const int b = k % (bins + 1);
            st[k] = b == bins ? 1.0 : (double)b / bins;
        }
    double* sc = st + D * (bins + 1);
    for (int k = threadIdx.x; k < kStSlots; k += blockDim.x) sc[k] = 0.0;
}

// ===========================================================================
// launchers

template <typename T, int TERM>
cudaError_t launch_points_t(const void* args, const InnerRule& rule, const double* x, int64_t n, double* out,
                            cudaStream_t stream)
{
    // A nested FP32 term evaluates the points of a warp one after the other, all lanes on the nodes of
    // one: as few points a warp as the resident warps (8 CTAs of 4 per SM) take in one pass, a power
    // of two.  200 points with 16 and 48 nodes: 6.1 and 7.0 us, 21.2 and 35.7 with 32 points a warp
    // (13.1 and 31.2 with a lane per point); 10,000: 10.7 and 14.0, 21.5 and 36.5 (14.1 and 34.0).
    int per_warp = 32;
    if constexpr (warp_term<T, TERM>()) {
        int device = 0, sms = 148;
        if (cudaGetDevice(&device) == cudaSuccess)
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        while (per_warp > 1 && n * 2 <= (int64_t)sms * 32 * per_warp) per_warp /= 2;
    }
    const int64_t per_cta = (int64_t)per_warp * (kPointsThreads / 32);
    int64_t blocks = (n + per_cta - 1) / per_cta;
    blocks = blocks > 4096 ? 4096 : (blocks < 1 ? 1 : blocks);
    points_kernel<T, TERM><<<(unsigned)blocks, kPointsThreads, 0, stream>>>(*static_cast<const DisArgs<T>*>(args), rule, x, n,
                                                                     per_warp, out);
    return cudaGetLastError();
}

template <typename T, int TERM>
cudaError_t launch_gl_t(const void* args, int jobs, const InnerRule& rule, const GLRules& gl, double* out,
                        cudaStream_t stream)
{
    if constexpr (term_dims(TERM) == 2) {
        gauss_legendre_kernel<T, TERM><<<jobs, 256, 0, stream>>>(static_cast<const DisArgs<T>*>(args), rule, gl, out);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <typename T, int TERM>
cudaError_t launch_vegas_round_t(const VegasLaunch& L, cudaStream_t stream)
{
    constexpr int D = term_dims(TERM);
    const size_t smem = (sizeof(double2) + sizeof(double) * (kVegasThreads / 32) + sizeof(int32_t)) * D * (size_t)L.bins;
    auto kern = vegas_iteration_kernel<T, TERM>;
    cudaError_t e = raise_dynamic_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    dim3 grid(L.blocks_per_job, L.jobs);
    kern<<<grid, kVegasThreads, smem, stream>>>(static_cast<const DisArgs<T>*>(L.args), L.dirs, *L.rule, L.state,
                                                L.state_stride, L.bins, L.offset, L.samples, L.blocks_per_job,
                                                L.partial, L.counts);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int keys = 2 + D * L.bins;
    dim3 rgrid((keys + kReduceKeys - 1) / kReduceKeys, L.jobs);
    vegas_reduce_kernel<<<rgrid, kReduceKeys * kReduceSlices, 0, stream>>>(L.partial, keys, L.blocks_per_job,
                                                                           L.reduced);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t fsmem = sizeof(double) * (D * L.bins + 2 * D * (L.bins + 1));
    e = raise_dynamic_smem((const void*)vegas_finalize_kernel, fsmem);
    if (e != cudaSuccess) return e;
    vegas_finalize_kernel<<<L.jobs, 256, fsmem, stream>>>(L.state, L.state_stride, D, L.bins, L.samples, L.reduced,
                                                          L.counts, L.warmup, L.min_iterations, L.epsrel, L.epsabs);
    return cudaGetLastError();
}

#define NLO_DIS_DISPATCH(FN, ...)                                                  \
    switch (term) {                                                                \
        case kTermLO: return FN<T, kTermLO>(__VA_ARGS__);                          \
        case kTermDip0: return FN<T, kTermDip0>(__VA_ARGS__);                      \
        case kTermDip1: return FN<T, kTermDip1>(__VA_ARGS__);                      \
        case kTermDip2: return FN<T, kTermDip2>(__VA_ARGS__);                      \
        case kTermI1: return FN<T, kTermI1>(__VA_ARGS__);                          \
        case kTermI2: return FN<T, kTermI2>(__VA_ARGS__);                          \
        case kTermI3: return FN<T, kTermI3>(__VA_ARGS__);                          \
        case kTermI2N: return FN<T, kTermI2N>(__VA_ARGS__);                        \
        case kTermI3N: return FN<T, kTermI3N>(__VA_ARGS__);                        \
        default: return cudaErrorInvalidValue;                                     \
    }

template <typename T>
cudaError_t launch_points_typed(int term, const void* args, const InnerRule& rule, const double* x, int64_t n,
                                double* out, cudaStream_t stream)
{
    NLO_DIS_DISPATCH(launch_points_t, args, rule, x, n, out, stream)
}

template <typename T>
cudaError_t launch_gl_typed(int term, const void* args, int jobs, const InnerRule& rule, const GLRules& gl,
                            double* out, cudaStream_t stream)
{
    switch (term) {
        case kTermLO: return launch_gl_t<T, kTermLO>(args, jobs, rule, gl, out, stream);
        case kTermDip0: return launch_gl_t<T, kTermDip0>(args, jobs, rule, gl, out, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t launch_vegas_round_typed(int term, const VegasLaunch& L, cudaStream_t stream)
{
    NLO_DIS_DISPATCH(launch_vegas_round_t, L, stream)
}

}  // namespace dis

cudaError_t dis_launch_table_prepare(const double* r, const double* y, const double* N, int nr, int ny, double y0,
                                     int interp, double* table, cudaStream_t stream)
{
    int blocks = (nr * ny + 255) / 256;
    blocks = blocks > 1024 ? 1024 : (blocks < 1 ? 1 : blocks);
    dis::table_prepare_kernel<<<blocks, 256, 0, stream>>>(r, y, N, nr, ny, y0, interp, table);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    int64_t items = (int64_t)ny * (nr - 1);
    int64_t local_blocks = (items + 255) / 256;
    local_blocks = local_blocks > 2048 ? 2048 : (local_blocks < 1 ? 1 : local_blocks);
    dis::table_local_kernel<<<(unsigned)local_blocks, 256, 0, stream>>>(table, nr, ny);
    return cudaGetLastError();
}

cudaError_t dis_launch_table_initialize(double* table, int nr, int ny, double Y, cudaStream_t stream)
{
    const size_t smem = sizeof(double) * 3 * (size_t)nr;
    cudaError_t e = raise_dynamic_smem((const void*)dis::table_initialize_kernel, smem);
    if (e != cudaSuccess) return e;
    dis::table_initialize_kernel<<<1, 256, smem, stream>>>(table, nr, ny, Y);
    return cudaGetLastError();
}

cudaError_t dis_launch_points(int precision, int term, const void* args, const dis::InnerRule& rule, const double* x,
                              int64_t n, double* out, cudaStream_t stream)
{
    return precision == NLO_PRECISION_FP64 ? dis::launch_points_typed<double>(term, args, rule, x, n, out, stream)
                                           : dis::launch_points_typed<float>(term, args, rule, x, n, out, stream);
}

cudaError_t dis_launch_amplitude(int precision, const void* args, const double* r, const double* Y, int64_t n,
                                 double* out, cudaStream_t stream)
{
    int64_t blocks = (n + 255) / 256;
    blocks = blocks > 4096 ? 4096 : (blocks < 1 ? 1 : blocks);
    if (precision == NLO_PRECISION_FP64)
        dis::amplitude_kernel<double><<<(unsigned)blocks, 256, 0, stream>>>(
            *static_cast<const dis::DisArgs<double>*>(args), r, Y, n, out);
    else
        dis::amplitude_kernel<float><<<(unsigned)blocks, 256, 0, stream>>>(
            *static_cast<const dis::DisArgs<float>*>(args), r, Y, n, out);
    return cudaGetLastError();
}

cudaError_t dis_launch_gl(int precision, int term, const void* args, int jobs, const dis::InnerRule& rule,
                          const dis::GLRules& gl, double* out, cudaStream_t stream)
{
    return precision == NLO_PRECISION_FP64 ? dis::launch_gl_typed<double>(term, args, jobs, rule, gl, out, stream)
                                           : dis::launch_gl_typed<float>(term, args, jobs, rule, gl, out, stream);
}

cudaError_t dis_launch_vegas_init(double* state, int state_stride, int D, int bins, int jobs, int keep_edges,
                                  int32_t* counts, cudaStream_t stream)
{
    dis::vegas_init_kernel<<<jobs, 128, 0, stream>>>(state, state_stride, D, bins, jobs, keep_edges, counts);
    return cudaGetLastError();
}

cudaError_t dis_launch_reduce_finalize(int D, int bins, int jobs, int blocks_per_job, const double* partial,
                                       double* reduced, int32_t* counts, double* state, int state_stride,
                                       uint64_t samples, int warmup, int min_iterations, double epsrel, double epsabs,
                                       cudaStream_t stream)
{
    const int keys = 2 + D * bins;
    dim3 rgrid((keys + dis::kReduceKeys - 1) / dis::kReduceKeys, jobs);
    dis::vegas_reduce_kernel<<<rgrid, dis::kReduceKeys * dis::kReduceSlices, 0, stream>>>(partial, keys,
                                                                                       blocks_per_job, reduced);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t fsmem = sizeof(double) * (D * bins + 2 * D * (bins + 1));
    e = raise_dynamic_smem((const void*)dis::vegas_finalize_kernel, fsmem);
    if (e != cudaSuccess) return e;
    dis::vegas_finalize_kernel<<<jobs, 256, fsmem, stream>>>(state, state_stride, D, bins, samples, reduced, counts,
                                                               warmup, min_iterations, epsrel, epsabs);
    return cudaGetLastError();
}

cudaError_t vegas_launch_reduce(const double* partial, int keys, int blocks_per_job, int jobs, double* reduced,
                                cudaStream_t stream)
{
    dim3 rgrid((keys + dis::kReduceKeys - 1) / dis::kReduceKeys, jobs);
    dis::vegas_reduce_kernel<<<rgrid, dis::kReduceKeys * dis::kReduceSlices, 0, stream>>>(partial, keys,
                                                                                       blocks_per_job, reduced);
    return cudaGetLastError();
}

cudaError_t dis_launch_vegas_round(int precision, int term, const dis::VegasLaunch& L, cudaStream_t stream)
{
    return precision == NLO_PRECISION_FP64 ? dis::launch_vegas_round_typed<double>(term, L, stream)
                                           : dis::launch_vegas_round_typed<float>(term, L, stream);
}

}  // namespace nlo
