/*
 * Sweeps and measurements of one lattice in global memory, L_x a multiple of
 * 4, walked along z in patches (walk_global.cuh): the single-task calls and the
 * large lattices of a batch.
 *
 *   k_walk_colour   one colour of metropolis_sweep_with_scratch
 *                   (src/updates.rs:440-486); colour 0 optionally fused with
 *                   the measurement of the state it starts from
 *   k_walk_measure  measure_theta_observables_with_scratch
 *                   (src/observables.rs:80-154)
 */
#include <algorithm>

#include "engine.h"
#include "walk_global.cuh"

namespace slsf {

namespace {

constexpr int kWalkThreads = 256;
constexpr int kWalkBlocksPerSm = 2; /* 128 registers a thread */

/* Adds a per-thread count to stats[slot] with one global atomic per block. */
__device__ __forceinline__ void block_count(uint32_t v, unsigned long long* stats, int slot) {
    __shared__ unsigned int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_sum, v);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(&stats[slot], (unsigned long long)s_sum);
}

/* The block's sums to the partials; the last block adds them in block order,
 * writes the totals and adds the measured values to bin_row (NULL: none). */
__device__ __forceinline__ void finish_sums(double (&acc)[8], const TaskView& t, double* bin_row) {
    __shared__ double scratch[8 * 32];
    __shared__ bool last;
    block_sum<8>(acc, scratch);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) t.partials[blockIdx.x * 8 + k] = acc[k];
        __threadfence();
        last = atomicAdd(t.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < 8; ++k) tot[k] += __ldcg(&t.partials[b * 8 + k]);
    block_sum<8>(tot, scratch);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) t.result[k] = tot[k];
        if (bin_row) add_to_bin(t, tot, bin_row);
        *t.done = 0;
    }
}

/* One colour.  Bound by instruction issue and the special-function pipe (two
 * Philox blocks, 14 neighbour and 8 own sincos per four updates: 53 and 52% of
 * their cycles); angles come from L2 or HBM, 12 bytes per update.  At L = 256
 * 41 us, 82 with the measurement (one thread per Philox block: 70 and 115). */
template <bool kMeasure>
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocksPerSm)
    k_walk_colour(TaskView t, uint64_t sweep, uint32_t colour, uint32_t seglen, double* bin_row) {
    WalkSums sums;
    if (kMeasure) sums.start(t.jxy_max, t.jz_max);
    const uint32_t accepted = walk_colour<kMeasure>(t, sweep, colour, seglen, blockIdx.x * kWalkThreads + threadIdx.x, &sums);
    block_count(accepted, t.stats, kStatAccepted);
    if (kMeasure) finish_sums(sums.acc, t, bin_row);
}

/* The observables of the state: 14 sincos per eight sites.  The terms gathered
 * in FP32 value and remainder (Sum2) instead of an FP64 conversion each on the
 * special-function pipe, which bound the earlier row walk (72% of it busy, 86
 * us at L = 256; now 45% and 52 us). */
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocksPerSm)
    k_walk_measure(TaskView t, uint32_t seglen, double* bin_row) {
    WalkSums sums;
    sums.start(t.jxy_max, t.jz_max);
    walk_measure(t, seglen, blockIdx.x * kWalkThreads + threadIdx.x, sums);
    finish_sums(sums.acc, t, bin_row);
}

uint32_t walk_blocks(const TaskView& t, uint32_t seglen) {
    return (walk_units(t, seglen) + kWalkThreads - 1) / kWalkThreads;
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

bool walk_supports(const TaskView& t) {
    /* patches of four sites by two rows; the biased runs need finite couplings; 32-bit site indices; a block sum per
     * block of the partials' rows */
    return t.lx % 4 == 0 && t.ly % 2 == 0 && t.lz >= 2 && fmaxf(t.jxy_max, t.jz_max) < kJMax &&
           (reinterpret_cast<uintptr_t>(t.theta) & 15u) == 0 && (uint64_t)t.lx * t.ly * t.lz <= 0x7fffffffull &&
           walk_blocks(t, t.lz) <= (uint32_t)kMeasureMaxBlocks;
}

static uint32_t walk_seglen(const TaskView& t) {
    /* Planes per thread: as many segments as fill one, two, three or four
     * rounds of the resident blocks, whichever ends first when a round takes its
     * planes and about 0.7 of a plane to fill the window; at least two planes.
     * (L = 256: 29 planes, 288 blocks on 296 places; L = 64: two, 64 blocks.) */
    const uint64_t places = (uint64_t)sm_count() * kWalkBlocksPerSm, ncol = (uint64_t)(t.lx >> 2) * (t.ly >> 1);
    uint32_t best = t.lz;
    double cost = 1e300;
    for (uint32_t r = 1; r <= 4; ++r) {
        const uint64_t blocks = std::min<uint64_t>(std::max<uint64_t>(r * places, 1), kMeasureMaxBlocks);
        const uint64_t nseg = std::min<uint64_t>(std::max<uint64_t>(blocks * kWalkThreads / ncol, 1), std::max(1u, t.lz / 2));
        const uint32_t len = (uint32_t)((t.lz + nseg - 1) / nseg);
        const double rounds = (double)((walk_blocks(t, len) + places - 1) / places);
        if (rounds * (len + 0.7) < cost) {
            cost = rounds * (len + 0.7);
            best = len;
        }
    }
    return best;
}

void launch_walk_colour(const TaskView& t, uint64_t sweep, uint32_t colour, bool measure, double* bin_row, cudaStream_t s) {
    const uint32_t len = walk_seglen(t);
    if (measure)
        k_walk_colour<true><<<walk_blocks(t, len), kWalkThreads, 0, s>>>(t, sweep, colour, len, bin_row);
    else
        k_walk_colour<false><<<walk_blocks(t, len), kWalkThreads, 0, s>>>(t, sweep, colour, len, nullptr);
}

void launch_walk_measure(const TaskView& t, double* bin_row, cudaStream_t s) {
    const uint32_t len = walk_seglen(t);
    k_walk_measure<<<walk_blocks(t, len), kWalkThreads, 0, s>>>(t, len, bin_row);
}

}  // namespace slsf
