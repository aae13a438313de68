/*
 * Single-task Wolff update on bit-packed bonds: grows the seed's cluster
 * only, for lattices whose three sides are multiples of 32 (the large
 * single-replica lattices: L = 64 ... 256 and more).
 *
 * Replaces, for those shapes, the whole-lattice union-find labelling of
 * kernels_plain.cu.  The reference grows one cluster from a random seed by
 * depth-first search (wolff_cluster_step_with_theta_scratch,
 * src/updates.rs:551-620); with one counter-based random per bond, that
 * cluster is the seed's connected component over the active bonds, and only
 * it is needed.
 *
 *   k_wb_bonds   per-site +x/+y/+z bond activation (try_add_wolff_neighbor,
 *                src/updates.rs:537-548) into three bit planes: bit i of the
 *                flat bitmap is site i (site index x + Lx (y + Ly z), so a
 *                32-bit word is 32 consecutive sites of one row); clears the
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
#include "wolff_global.cuh"
#include "xy_device.cuh"

namespace slsf {

namespace {

constexpr uint32_t kRegion = kGrowEdge; /* region edge in sites along y and z; one word along x */
constexpr uint32_t kGrowThreads = kRegion * kRegion;
constexpr int kBondThreads = 256;
constexpr int kFlipThreads = 256;
constexpr int kFlipQuads = 4; /* quads of sites per thread */
constexpr uint32_t kEmpty = 0;
constexpr uint32_t kNoRegion = 0xffffffffu;

/* Optional counters (build with -DSLSF_WB_STATS): regions processed, growth
 * passes, grow launches, and region loads that changed nothing. */
#ifdef SLSF_WB_STATS
/* [0] regions processed, [1] passes, [2] grow launches, [3] loads without new
 * bits, [4..7] cycles of thread 0 in: waiting for work, loading, closing,
 * writing back and queueing neighbours */
__device__ unsigned long long g_wb_stats[8];
#define SLSF_WB_CLOCK(k, t0)                                                                     \
    do {                                                                                         \
        if (threadIdx.x == 0) {                                                                  \
            const long long t1_ = clock64();                                                     \
            atomicAdd(&g_wb_stats[k], (unsigned long long)(t1_ - (t0)));                         \
            (t0) = t1_;                                                                          \
        }                                                                                        \
    } while (0)
#define SLSF_WB_COUNT(k, n)                                                          \
    do {                                                                             \
        if (threadIdx.x == 0) atomicAdd(&g_wb_stats[k], (unsigned long long)(n));    \
    } while (0)
#else
#define SLSF_WB_COUNT(k, n) \
    do {                    \
    } while (0)
#define SLSF_WB_CLOCK(k, t0) \
    do {                     \
    } while (0)
#endif

/* Scratch of one update, carved from the task's union-find array. */
struct WolffBits {
    uint32_t* bx;      /* bond bit planes, one bit per site */
    uint32_t* by;
    uint32_t* bz;
    uint32_t* cl;      /* cluster bitmap */
    uint32_t* queued;  /* [regions] 1 while the region is in the queue */
    uint32_t* ring;    /* [cap] region + 1, or 0 */
    uint32_t* ctl;     /* head, tail, pending (queued or in flight), abort, seed site + 1 */
    uint32_t regions, cap;
};

__host__ __device__ inline uint64_t round256(uint64_t b) { return (b + 255) & ~255ull; }

__host__ __device__ inline uint64_t bit_words(uint32_t lx, uint32_t ly, uint32_t lz) {
    return (uint64_t)((lx + 31) / 32) * ly * lz;
}

__host__ __device__ inline uint64_t bit_regions(uint32_t lx, uint32_t ly, uint32_t lz) {
    return (uint64_t)((lx + 31) / 32) * ((ly + kRegion - 1) / kRegion) * ((lz + kRegion - 1) / kRegion);
}

__host__ __device__ inline uint64_t pow2_at_least(uint64_t n) {
    uint64_t p = 1;
    while (p < n) p <<= 1;
    return p;
}

__host__ __device__ inline uint64_t control_bytes(uint64_t regions) {
    return round256(4 * regions) + round256(4 * pow2_at_least(2 * regions + 2)) + 256;
}

/* The scratch of one update: bit planes, then the control words (queued, ring, ctl; zero at its start). */
__host__ __device__ inline WolffBits carve_bits(void* scratch, uint32_t lx, uint32_t ly, uint32_t lz) {
    const uint64_t plane = round256(4 * bit_words(lx, ly, lz)) / 4;
    uint32_t* p = static_cast<uint32_t*>(scratch);
    WolffBits wb;
    wb.bx = p;
    wb.by = p + plane;
    wb.bz = p + 2 * plane;
    wb.cl = p + 3 * plane;
    wb.regions = (uint32_t)bit_regions(lx, ly, lz);
    wb.cap = (uint32_t)pow2_at_least(2ull * wb.regions + 2);
    wb.queued = p + 4 * plane;
    wb.ring = wb.queued + round256(4ull * wb.regions) / 4;
    wb.ctl = wb.ring + round256(4ull * wb.cap) / 4;
    return wb;
}


/* Makes the seed's region the first queue entry (the control words are zero). */
__device__ __forceinline__ void queue_seed(const WolffBits& wb, uint32_t lx, uint32_t ly, uint32_t lz, uint32_t x, uint32_t y,
                                           uint32_t z) {
    const uint32_t words = (lx + 31u) >> 5;
    const uint32_t r = (x >> 5) + words * ((y / kRegion) + ((ly + kRegion - 1) / kRegion) * (z / kRegion));
    wb.queued[r] = 1;
    wb.ring[0] = r + 1;
    wb.ctl[1] = 1; /* tail */
    wb.ctl[2] = 1; /* pending */
    wb.ctl[4] = x + lx * (y + ly * z) + 1; /* the seed's bit enters its region like a face bit */
}

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

struct GrowGeo {
    uint32_t lx, ly, lz, words, ry_n, rz_n;
    bool px, py, pz; /* the region spans the whole period along x (one-word rows), y (32 rows), z (32 planes) */
};

__host__ __device__ inline GrowGeo grow_geo(uint32_t lx, uint32_t ly, uint32_t lz) {
    return {lx, ly, lz, (lx + 31) / 32, (ly + kRegion - 1) / kRegion, (lz + kRegion - 1) / kRegion,
            lx <= 32, ly == kRegion, lz == kRegion};
}

/* Claims region r for processing unless it is claimed already (queued or
 * kept): the first neighbour a CTA claims it keeps in *keep and processes
 * next itself, the others go to the queue. */
__device__ __forceinline__ void push_region(const WolffBits& wb, uint32_t r, uint32_t* keep) {
    if (atomicExch(&wb.queued[r], 1u) != 0u) return;
    atomicAdd(&wb.ctl[2], 1u); /* pending before the region can be taken */
    if (atomicCAS(keep, kNoRegion, r) == kNoRegion) return;
    const uint32_t slot = atomicAdd(&wb.ctl[1], 1u);
    __threadfence();
    atomicExch(&wb.ring[slot & (wb.cap - 1)], r + 1);
}

__device__ __forceinline__ uint32_t region_of(const GrowGeo& g, uint32_t k, uint32_t ry, uint32_t rz) {
    return k + g.words * (ry + g.ry_n * rz);
}

/* One region: load with the bits entering through its faces, close in
 * shared memory, OR back, queue the neighbours its bits can enter.  Returns
 * false if a pass bound was hit. */
__device__ bool grow_region(const WolffBits& wb, const GrowGeo& g, uint32_t r, uint32_t seed_word, uint32_t seed_bit,
                            uint32_t (*C)[kRegion + 1], uint32_t (*BY)[kRegion + 1], uint32_t (*BZ)[kRegion + 1],
                            uint32_t (*BX)[kRegion + 1], uint32_t* keep, uint32_t* s_want) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t k = r % g.words, rest = r / g.words, ry = rest % g.ry_n, rz = rest / g.ry_n;
    const uint32_t rowlen = g.words; /* words per row */
    const uint32_t gy = ry * kRegion + lane, gz = rz * kRegion + warp;
    /* rows and planes past the lattice hold zeros; the last ones of a region face the next region */
    const bool in = gy < g.ly && gz < g.lz;
    const bool last_y = lane == kRegion - 1 || gy + 1 == g.ly, last_z = warp == kRegion - 1 || gz + 1 == g.lz;
    /* the word's last site, and that of the word to its left */
    const uint32_t top = min(32u, g.lx - 32u * k) - 1, kl = k == 0 ? g.words - 1 : k - 1;
    const uint32_t top_l = min(32u, g.lx - 32u * kl) - 1;
    auto word = [&](uint32_t kk, uint32_t yy, uint32_t zz) { return kk + rowlen * (yy + g.ly * zz); };
#ifdef SLSF_WB_STATS
    long long tclk = clock64();
#endif
    const uint32_t w = in ? word(k, gy, gz) : 0u;
    /* the region's own words (written only by processings of this region) */
    const uint32_t c0 = in ? __ldcg(&wb.cl[w]) : 0u;
    const uint32_t bxw = in ? wb.bx[w] : 0u, byw = in ? wb.by[w] : 0u, bzw = in ? wb.bz[w] : 0u;
    /* claimable again from here on: the reset is visible before the
     * neighbours' words are read, so a neighbour that adds face bits later
     * finds the region unqueued and queues it */
    if (threadIdx.x == 0) {
        wb.queued[r] = 0u;
        __threadfence();
    }
    __syncthreads();
    uint32_t c = c0;
    /* bits entering through the faces */
    const uint32_t kr = k + 1 == g.words ? 0 : k + 1;
    const uint32_t ym = gy == 0 ? g.ly - 1 : gy - 1, yp = gy + 1 == g.ly ? 0 : gy + 1;
    const uint32_t zm = gz == 0 ? g.lz - 1 : gz - 1, zp = gz + 1 == g.lz ? 0 : gz + 1;
    /* the faces' neighbour words as loaded here also decide, at the end,
     * which neighbours to queue: a neighbour word only ever gains bits, so a
     * stale copy can queue a region that needs nothing, never miss one */
    uint32_t cl_l = ~0u, bx_l = 0, cl_r = ~0u, cl_ym = ~0u, by_ym = 0, cl_yp = ~0u, cl_zm = ~0u, bz_zm = 0, cl_zp = ~0u;
    if (!g.px && in) {
        const uint32_t wl = word(kl, gy, gz), wr = word(kr, gy, gz);
        cl_l = __ldcg(&wb.cl[wl]);
        bx_l = wb.bx[wl];
        cl_r = __ldcg(&wb.cl[wr]);
        c |= (cl_l >> top_l) & (bx_l >> top_l) & 1u;
        c |= ((cl_r & 1u) & (bxw >> top)) << top;
    }
    if (!g.py && in) {
        if (lane == 0) {
            const uint32_t wm = word(k, ym, gz);
            cl_ym = __ldcg(&wb.cl[wm]);
            by_ym = wb.by[wm];
            c |= cl_ym & by_ym;
        }
        if (last_y) {
            cl_yp = __ldcg(&wb.cl[word(k, yp, gz)]);
            c |= cl_yp & byw;
        }
    }
    if (!g.pz && in) {
        if (warp == 0) {
            const uint32_t wm = word(k, gy, zm);
            cl_zm = __ldcg(&wb.cl[wm]);
            bz_zm = wb.bz[wm];
            c |= cl_zm & bz_zm;
        }
        if (last_z) {
            cl_zp = __ldcg(&wb.cl[word(k, gy, zp)]);
            c |= cl_zp & bzw;
        }
    }
    if (in && seed_word == w) c |= 1u << seed_bit;
    /* inside the word: bond bit `top` of an open word leads out of it */
    const uint32_t bxi = g.px ? bxw : bxw & ((1u << top) - 1u);
    c = g.px ? close_word(c, bxi, g.lx, true) : close_word(c, bxi, 32u, false);
    /* the stored region is closed already: without new bits nothing changes */
    const int any_new = __syncthreads_or(c != c0);
    SLSF_WB_CLOCK(5, tclk);
    if (!any_new) {
        SLSF_WB_COUNT(3, 1);
        return true;
    }
    C[warp][lane] = c;
    BX[warp][lane] = bxi;
    BY[warp][lane] = last_y && !g.py ? 0u : byw; /* the bonds out of the region are the faces' */
    BZ[warp][lane] = last_z && !g.pz ? 0u : bzw;
    __syncthreads();
    const GrowBlock q = {&C[0][0], &BX[0][0], &BY[0][0], &BZ[0][0], g.px ? g.lx : 32u, g.px, g.py, g.pz};
    const uint32_t passes = close_block(q, kRegion * kRegion * kRegion + 1);
    SLSF_WB_COUNT(1, passes);
    SLSF_WB_CLOCK(6, tclk);
    const bool ok = passes != 0;
    c = C[warp][lane];
    if (in && c != c0) atomicOr(&wb.cl[w], c);
    /* neighbours that the region's bits can enter: bit 0/1 -x/+x, 2/3 -y/+y, 4/5 -z/+z */
    uint32_t want = 0;
    if (!g.px && in) {
        if ((c & 1u) && (bx_l >> top_l & 1u) && !(cl_l >> top_l & 1u)) want |= 1u;
        if ((c >> top & 1u) && (bxw >> top & 1u) && !(cl_r & 1u)) want |= 2u;
    }
    if (!g.py && in) {
        if (lane == 0 && (c & by_ym & ~cl_ym)) want |= 4u;
        if (last_y && (c & byw & ~cl_yp)) want |= 8u;
    }
    if (!g.pz && in) {
        if (warp == 0 && (c & bz_zm & ~cl_zm)) want |= 16u;
        if (last_z && (c & bzw & ~cl_zp)) want |= 32u;
    }
    want = __reduce_or_sync(0xffffffffu, want);
    if (lane == 0 && want) atomicOr(s_want, want);
    __syncthreads();
    /* thread d queues the neighbour in direction d, so that the six queue
     * operations (each a few dependent atomics) overlap; the block's cluster
     * words are written (barrier above) and each pushing thread's fence
     * orders them before its neighbour can be taken */
    const uint32_t m = *s_want;
    if (threadIdx.x < 6 && ((m >> threadIdx.x) & 1u)) {
        uint32_t nb;
        switch (threadIdx.x) {
            case 0: nb = region_of(g, k == 0 ? g.words - 1 : k - 1, ry, rz); break;
            case 1: nb = region_of(g, k + 1 == g.words ? 0 : k + 1, ry, rz); break;
            case 2: nb = region_of(g, k, ry == 0 ? g.ry_n - 1 : ry - 1, rz); break;
            case 3: nb = region_of(g, k, ry + 1 == g.ry_n ? 0 : ry + 1, rz); break;
            case 4: nb = region_of(g, k, ry, rz == 0 ? g.rz_n - 1 : rz - 1); break;
            default: nb = region_of(g, k, ry, rz + 1 == g.rz_n ? 0 : rz + 1); break;
        }
        __threadfence();
        push_region(wb, nb, keep);
    }
    __syncthreads(); /* every thread has read the mask before it is cleared */
    if (threadIdx.x == 0) *s_want = 0;
    return ok;
}

/* Takes regions until nothing is queued or in flight. */
__device__ __forceinline__ void grow_regions(const WolffBits& wb, const GrowGeo& g, uint32_t max_items,
                                             unsigned long long* __restrict__ stats) {
    __shared__ uint32_t C[kRegion][kRegion + 1];
    __shared__ uint32_t BY[kRegion][kRegion + 1];
    __shared__ uint32_t BZ[kRegion][kRegion + 1];
    __shared__ uint32_t BX[kRegion][kRegion + 1];
    __shared__ uint32_t s_item;
    __shared__ uint32_t s_keep;
    __shared__ uint32_t s_want;
    /* Each CTA takes regions until nothing is queued or in flight: the
     * neighbour it claimed while processing the last one (no queue round
     * trip), else the queue entry of its ticket (one atomic; the producer
     * may not have filled it yet, the CTA waits for it, bounded).  A ticket
     * whose entry never comes is given up when nothing is pending. */
    constexpr uint32_t kSpin = 1u << 24;
    const uint32_t seed_site = __ldcg(&wb.ctl[4]) - 1, seed_row = seed_site / g.lx, seed_x = seed_site - seed_row * g.lx;
    const uint32_t seed_word = seed_row * g.words + (seed_x >> 5), seed_bit = seed_x & 31u;
    bool ok = true;
    if (threadIdx.x == 0) {
        s_keep = kNoRegion;
        s_want = 0;
    }
    __syncthreads();
#ifdef SLSF_WB_STATS
    long long tq = clock64();
#endif
    for (uint32_t item = 0; item < max_items; ++item) {
        if (threadIdx.x == 0) {
#ifdef SLSF_WB_STATS
            tq = clock64();
#endif
            uint32_t got = s_keep;
            if (got == kNoRegion) {
                got = 0xfffffffeu; /* gave up, unless set below */
                const uint32_t ticket = atomicAdd(&wb.ctl[0], 1u);
                volatile uint32_t* slot = &wb.ring[ticket & (wb.cap - 1)];
                volatile uint32_t* ctl = wb.ctl;
                for (uint32_t spin = 0; spin < kSpin; ++spin) {
                    const uint32_t v = *slot;
                    if (v != kEmpty) {
                        *slot = kEmpty;
                        got = v - 1;
                        break;
                    }
                    if (ctl[2] == 0 || ctl[3] != 0) { /* nothing queued or in flight, or aborted */
                        got = 0xffffffffu;
                        break;
                    }
                    __nanosleep(32);
                }
            }
            s_keep = kNoRegion;
            s_item = got;
        }
        __syncthreads();
        SLSF_WB_CLOCK(4, tq);
        const uint32_t r = s_item;
        if (r == 0xffffffffu) break;
        if (r >= wb.regions) {
            ok = false;
            break;
        }
        ok &= grow_region(wb, g, r, seed_word, seed_bit, C, BY, BZ, BX, &s_keep, &s_want);
        SLSF_WB_COUNT(0, 1);
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicSub(&wb.ctl[2], 1u);
        }
        SLSF_WB_CLOCK(7, tq);
        if (item + 1 == max_items) ok = false;
    }
    if (!ok && threadIdx.x == 0) {
        atomicOr(&stats[kStatError], kErrGrowthLimit);
        atomicExch(&wb.ctl[3], 1u); /* the other CTAs stop at their next pop */
    }
}

__global__ void __launch_bounds__(kGrowThreads, 1)
    k_wb_grow(WolffBits wb, GrowGeo g, uint32_t max_items, unsigned long long* __restrict__ stats) {
    grow_regions(wb, g, max_items, stats);
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
