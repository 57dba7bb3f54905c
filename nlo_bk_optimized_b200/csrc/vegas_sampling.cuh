// Warp-level sampling pieces of the device Vegas rounds (dis.cu, k2kf_vegas.cu).
//
// A warp takes 32 consecutive Sobol points at a time, starting at a multiple of 32.  Two
// properties of such a block carry the code below:
//
// * gray(32 k + l) = gray(32 k) ^ gray(l) for l < 32, so a point's bits are the xor of a part of
//   the lane alone and a part of the block alone, and the block's part is one warp reduction
//   (lane j contributes direction number j) instead of a loop over the set bits in every lane;
// * in each dimension the 32 points fall into the 32 intervals of length 1/32, one each (a
//   digital net in base 2, which torch's scrambling preserves).  Two points can share a bin of a
//   grid only if few intervals lie between them, so a histogram needs `phases` conflict-free
//   additions (1 for bins = 32 or a multiple, 2 for any larger number) instead of matching
//   the lanes' bins.  Direction numbers that do not have the property (a caller's own), and the
//   block of point 0 (rounded to FP32 by torch), take one phase per lane.
//
// Both orders are fixed, so the sums are reproducible.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nlo {
namespace vegas {

// Per CTA: the direction numbers of D dimensions (rows past 29 are zero) and every lane's own
// part of the xor, [D][32] each; shift and the number of phases per dimension.
template <int D>
struct SobolWarp {
    uint32_t dir[D][32], low[D][32], shift[D];
    int phases[D];
    bool even;  // 32 bins and a net in every dimension: a whole block counts once in every bin
};

// `state` and `shift` as in nlo_sobol_dirs; called by all threads of the CTA, before a
// barrier.
template <int D>
__device__ __forceinline__ void stage_sobol(SobolWarp<D>& s, const uint32_t (*state)[30], const uint32_t* shift,
                                            int bins)
{
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    if (threadIdx.x == 0) s.even = bins == 32;
    __syncthreads();
    for (int d = threadIdx.x >> 5; d < D; d += warps) {
        s.dir[d][lane] = lane < 30 ? state[d][lane] : 0u;
        const uint32_t g = lane ^ (lane >> 1);
        uint32_t v = 0;
#pragma unroll
        for (int j = 0; j < 5; ++j) v ^= (g >> j) & 1u ? state[d][j] : 0u;
        s.low[d][lane] = v;
        const bool net = __reduce_or_sync(0xffffffffu, 1u << (v >> 25)) == 0xffffffffu;
        if (lane == 0) {
            s.shift[d] = shift[d];
            s.phases[d] = !net ? 32 : bins % 32 == 0 ? 1 : (bins + 31) / bins + 1;
            if (!net) s.even = false;
        }
    }
}

// The 30 bits of dimension d of the lane's point of the block starting at `base` (a multiple of
// 32); point 0 as the float32 torch gives.
template <int D>
__device__ __forceinline__ uint32_t sobol_block_bits(const SobolWarp<D>& s, int d, uint32_t base)
{
    const int lane = threadIdx.x & 31;
    const uint32_t g = base ^ (base >> 1);
    const uint32_t block = __reduce_xor_sync(0xffffffffu, (g >> lane) & 1u ? s.dir[d][lane] : 0u);
    uint32_t bits = block ^ s.shift[d] ^ s.low[d][lane];
    if (base == 0 && lane == 0) bits = (uint32_t)__uint2float_rn(bits);
    return bits;
}

// Position of a coordinate u = bits 2^-30 in the grid: its bin, and 2^30 times the fraction within
// it (both exact).
__device__ __forceinline__ int grid_position(uint32_t bits, int bins, double& frac)
{
    const uint64_t scaled = (uint64_t)bits * (uint32_t)bins;
    int b = (int)(scaled >> 30);
    b = b > bins - 1 ? bins - 1 : b;
    const uint32_t rest = (uint32_t)(scaled - ((uint64_t)b << 30));
    // rest <= 2^30: 2^52 + rest holds it exactly
    frac = __hiloint2double(0x43300000, (int)rest) - 4503599627370496.0;
    return b;
}

// hist[bin] += value of the active lanes in every dimension, `hist` the warp's own rows
// [D][bins], and count[bin] += 1 in the CTA's; a whole block of an even grid only adds to `whole`,
// for add_whole_blocks.  All lanes call it; bits tell a lane's intervals of length 1/32.  The
// caller synchronises the CTA before the rows are read.
template <int D>
__device__ __forceinline__ void warp_hist_add(const SobolWarp<D>& s, uint32_t base, const uint32_t (&bits)[D],
                                              bool active, const int (&bin)[D], int bins, double value, double* hist,
                                              int32_t* count, int& whole)
{
    const bool counted = s.even && base != 0 && __all_sync(0xffffffffu, active);
    if (counted) ++whole;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const int phases = base == 0 ? 32 : s.phases[d];
        const int interval = (int)(bits[d] >> 25);
        double* h = hist + d * bins + bin[d];
        if (phases == 1) {
            if (active) *h += value;
        } else {
            const int mine = phases == 2 ? interval & 1 : phases == 32 ? (int)(threadIdx.x & 31) : interval % phases;
            for (int p = 0; p < phases; ++p) {
                if (active && mine == p) *h += value;
                __syncwarp();
            }
        }
        if (!counted && active) atomicAdd(&count[d * bins + bin[d]], 1);
    }
    // one phase: the next block's lanes find these additions (the dimensions' rows are disjoint)
    __syncwarp();
}

// The counts of a warp's whole blocks (32 bins: one per lane), before the barrier.
template <int D>
__device__ __forceinline__ void add_whole_blocks(int whole, int32_t* count)
{
    if (whole > 0)
        for (int d = 0; d < D; ++d) atomicAdd(&count[32 * d + (threadIdx.x & 31)], whole);
}

}  // namespace vegas
}  // namespace nlo
