/*
 * Single-task Wolff update on bit-packed bonds: grows the seed's cluster
 * only, for large single-replica lattices that are not too long for their size
 * (wolff_by_bits, kernels_plain.cu).
 *
 * Replaces, for those sizes, the whole-lattice union-find labelling of
 * kernels_plain.cu.  The reference grows one cluster from a random seed by
 * depth-first search (wolff_cluster_step_with_theta_scratch,
 * src/updates.rs:551-620); with one counter-based random per bond, that
 * cluster is the seed's connected component over the active bonds, and only
 * it is needed.
 *
 *   k_wb_bonds   per-site +x/+y/+z bond activation (try_add_wolff_neighbor,
 *                src/updates.rs:537-548) into three bit planes: bit x mod 32
 *                of word x / 32 of a row is site x, a row of L_x sites takes
 *                ceil(L_x / 32) words (wolff_global.cuh); clears the
 *                cluster bitmap and queues the seed's region, whose first
 *                processing adds the seed's bit.
 *   k_wb_grow    the cluster over the active bonds.  The lattice is cut into
 *                regions of 32 x 32 x 32 sites (one word wide, 32 rows, 32
 *                planes).  A CTA takes a region from a work queue, reads its
 *                cluster and bond words into shared memory with the bits that
 *                enter through the region's faces, closes the region in
 *                passes (each pass a full warp scan along y -- lane = y -- or
 *                along z -- lane = z, the shared array read transposed --
 *                one step along the other axis, and the closure along x
 *                inside each word), ORs the result back and queues every
 *                neighbour region its bits can enter.  Regions are processed
 *                as they are queued, with no grid-wide barrier: CTAs only
 *                wait for work that running CTAs hold, so the kernel needs
 *                no co-residency.  Bits only ever get set, so the fixed point
 *                is the seed's component whatever the order.
 *   k_wb_flip    reflection of the cluster's sites (src/updates.rs:602-617)
 *                and its size.
 *
 * Every wait and loop is bounded; past a bound the kernel sets
 * kErrGrowthLimit in the task's error word and returns.
 */
#include <algorithm>

#include "bitgrow.cuh"
#include "engine.h"
#include "fastdiv.h"
#include "region_grow.cuh"
#include "wolff_global.cuh"
#include "xy_device.cuh"

namespace slsf {

namespace {

constexpr int kBondThreads = 256;
constexpr int kFlipThreads = 256;
constexpr int kFlipQuads = 4; /* quads of sites per thread */

__global__ void __launch_bounds__(kBondThreads)
    k_wb_bonds(const float* __restrict__ theta, const float* __restrict__ jxy, const float* __restrict__ jz,
               uint32_t lx, uint32_t ly, uint32_t lz, float minus_two_beta, float phi, uint64_t seed,
               uint64_t counter, WolffBits wb, uint32_t seed_idx, uint32_t run, uint8_t* __restrict__ bond_bytes) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t row = seed_idx / lx;
        queue_seed(wb, lx, ly, lz, seed_idx - row * lx, row % ly, row / ly);
    }
    const BitPlanes planes = {wb.bx, wb.by, wb.bz, wb.cl};
    bond_run<1>(theta, jxy, jz, lx, ly, lz, minus_two_beta, phi, seed, counter, planes, run,
             (blockIdx.x * blockDim.x + threadIdx.x) >> 5, bond_bytes);
}

__global__ void __launch_bounds__(kGrowThreads, 1)
    k_wb_grow(WolffBits wb, GrowGeo g, uint32_t max_items, unsigned long long* __restrict__ stats) {
    grow_regions<1>(wb, g, max_items, stats);
}

/* Adds a per-thread count to stats[slot] with one global atomic per block. */
__device__ __forceinline__ void block_count(uint32_t n, unsigned long long* stats, int slot) {
    __shared__ unsigned int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&s_sum, n);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(&stats[slot], (unsigned long long)s_sum);
}

__global__ void __launch_bounds__(kFlipThreads)
    k_wb_flip(float* __restrict__ theta, uint32_t lx, uint32_t rows, slsf_fastdiv quads, const uint32_t* __restrict__ cl,
              float phi, unsigned long long* __restrict__ stats, uint8_t* __restrict__ cluster_out, bool wide) {
    block_count(flip_quads<kFlipQuads>(theta, lx, rows, blockIdx.x * kFlipQuads * blockDim.x + threadIdx.x, blockDim.x, quads, cl,
                                       phi, cluster_out, wide),
                stats, kStatClusterSites);
}

}  // namespace

uint64_t wolff_bits_scratch_bytes(uint32_t lx, uint32_t ly, uint32_t lz) {
    return 4 * round256(4 * bit_words(lx, ly, lz)) + control_bytes(bit_regions(lx, ly, lz));
}

int launch_wolff_bits(const TaskView& t, uint64_t counter, void* scratch, uint8_t* bond_bytes, uint8_t* cluster_out,
                      cudaStream_t s, float* phi_out, uint32_t seed_site[3]) {
    /* The reflection axis and seed site (src/updates.rs:564-568) from the
     * WOLFF_PICK block, computed on the host from the shared header. */
    const slsf_u32x4 pick = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_PICK, 0, 0);
    const float phi = slsf_angle_from_word(pick.x);
    const uint32_t x0 = slsf_range(pick.y, t.lx), y0 = slsf_range(pick.z, t.ly), z0 = slsf_range(pick.w, t.lz);
    const uint32_t volume = t.lx * t.ly * t.lz;
    const uint32_t seed_idx = x0 + t.lx * (y0 + t.ly * z0);
    const WolffBits wb = carve_bits(scratch, t.lx, t.ly, t.lz);
    cudaMemsetAsync(wb.queued, 0, control_bytes(wb.regions), s);
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    /* bond kernel: runs of rows per warp, halved while there are too few warps to give every SM a block's worth */
    const uint64_t cols = (uint64_t)((t.lx + 31) / 32) * ((t.lz + 1) / 2);
    uint32_t run = 32;
    while (run > 4 && cols * ((t.ly + run - 1) / run) < 16ull * (uint64_t)sms) run >>= 1;
    const uint64_t warps = cols * ((t.ly + run - 1) / run);
    const uint32_t bond_blocks = (uint32_t)((warps * 32 + kBondThreads - 1) / kBondThreads);
    k_wb_bonds<<<bond_blocks, kBondThreads, 0, s>>>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, -2.0f * t.beta, phi,
                                                    t.seed, counter, wb, seed_idx, run, bond_bytes);
    const GrowGeo g = grow_geo(t.lx, t.ly, t.lz);
    const uint32_t grid = std::min<uint32_t>(wb.regions, (uint32_t)sms);
    /* every region is processed at most once per bit it gains */
    const uint32_t max_items = t.loop_limit ? t.loop_limit : std::max<uint32_t>(64, volume / 32);
    k_wb_grow<<<grid, kGrowThreads, 0, s>>>(wb, g, max_items, t.stats);
    const slsf_fastdiv quads = slsf_fastdiv_make((t.lx + 3) / 4);
    const uint32_t rows = t.ly * t.lz;
    const bool wide = t.lx % 4 == 0 && (reinterpret_cast<uintptr_t>(t.theta) & 15u) == 0;
    k_wb_flip<<<(quads.d * rows + kFlipThreads * kFlipQuads - 1) / (kFlipThreads * kFlipQuads), kFlipThreads, 0, s>>>(
        t.theta, t.lx, rows, quads, wb.cl, phi, t.stats, cluster_out, wide);
    if (phi_out) *phi_out = phi;
    if (seed_site) {
        seed_site[0] = x0;
        seed_site[1] = y0;
        seed_site[2] = z0;
    }
    return 3;
}

}  // namespace slsf

#ifdef SLSF_WB_STATS
extern "C" int slsf_debug_wb_stats(unsigned long long out[8], int reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, slsf::g_wb_stats, sizeof(unsigned long long) * 8);
    if (e == cudaSuccess && reset) {
        const unsigned long long zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        e = cudaMemcpyToSymbol(slsf::g_wb_stats, zero, sizeof(zero));
    }
    return e == cudaSuccess ? 0 : 1;
}
#endif
