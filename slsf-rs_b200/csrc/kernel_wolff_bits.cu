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
#include "xy_device.cuh"

namespace slsf {

namespace {

constexpr uint32_t kRegion = kGrowEdge; /* region edge in sites along y and z; one word along x */
constexpr uint32_t kGrowThreads = kRegion * kRegion;
constexpr int kBondThreads = 256;
constexpr int kFlipThreads = 256;
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

/* Bond activation.  A warp owns word w (lane = bit = x - 32 w; lanes past the
 * row keep no bits) of the plane pair z, z + 1 for a run of up to 32 rows and
 * walks it along y, so the projections of the +y row are the next row's own
 * and plane z's +z partner is plane z + 1's site: three sincos for its two
 * sites, whose arithmetic is packed and whose Philox blocks share a key
 * schedule.  (The earlier walk of one plane took 186 instructions per site and
 * 133 us at L = 256.)  Lane j keeps the words of the run's row j and writes
 * them at its end.  With an odd L_z the last pair's second plane is plane 0,
 * computed and not kept.  The seed's region is queued. */
__global__ void __launch_bounds__(kBondThreads)
    k_wb_bonds(const float* __restrict__ theta, const float* __restrict__ jxy, const float* __restrict__ jz,
               uint32_t lx, uint32_t ly, uint32_t lz, float minus_two_beta, float phi, uint64_t seed,
               uint64_t counter, WolffBits wb, uint32_t seed_idx, uint32_t run, uint8_t* __restrict__ bond_bytes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t words = (lx + 31u) >> 5, nrun = (ly + run - 1) / run;
    const uint32_t w = wid % words, rest = wid / words;
    const uint32_t z = 2u * (rest / nrun), y_lo = (rest % nrun) * run;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        /* the seed's region is the first queue entry (the scratch was zeroed) */
        const uint32_t sx = seed_idx % lx, srow = seed_idx / lx, sy = srow % ly, sz = srow / ly;
        const uint32_t r = (sx >> 5) + words * ((sy / kRegion) + ((ly + kRegion - 1) / kRegion) * (sz / kRegion));
        wb.queued[r] = 1;
        wb.ring[0] = r + 1;
        wb.ctl[1] = 1; /* tail */
        wb.ctl[2] = 1; /* pending */
        wb.ctl[4] = seed_idx + 1; /* the seed's bit enters its region like a face bit */
    }
    if (z >= lz) return; /* whole warps */
    float sphi, cphi;
    __sincosf(phi, &sphi, &cphi);
    const float2 cphi2 = make_float2(cphi, cphi), sphi2 = make_float2(sphi, sphi);
    auto proj2 = [&](float a, float b) {
        float2 sn, cn;
        __sincosf(a, &sn.x, &cn.x);
        __sincosf(b, &sn.y, &cn.y);
        return __ffma2_rn(sn, sphi2, __fmul2_rn(cn, cphi2));
    };
    const uint32_t nv = min(32u, lx - 32u * w), rows = min(run, ly - y_lo);
    const uint32_t x = 32u * w + min(lane, nv - 1), xn = 32u * w + nv == lx ? 0u : 32u * w + 32u;
    const bool pair = z + 1 < lz;
    const uint32_t plane = lx * ly, z1 = pair ? z + 1 : 0u, z2 = z1 + 1 == lz ? 0u : z1 + 1;
    const float *p0 = theta + (size_t)z * plane, *p1 = theta + (size_t)z1 * plane, *p2 = theta + (size_t)z2 * plane;
    const float2 jx = make_float2(jxy[z], jxy[z1]), jzz = make_float2(jz[z], jz[z1]);
    const float2 m2b2 = make_float2(minus_two_beta, minus_two_beta);
    auto yrow = [&](uint32_t y) { return y + 1 == ly ? 0u : y + 1; };
    uint32_t o = y_lo * lx + x;
    float2 r = proj2(p0[o], p1[o]);
    /* lane j: the projections of the site after the word in row y_lo + j, the +x partner of the word's last site there */
    const uint32_t on = (y_lo + min(lane, rows - 1)) * lx + xn;
    const float2 r_next = proj2(p0[on], p1[on]);
    /* the angles of the next row's loads, one row ahead */
    uint32_t oy = yrow(y_lo) * lx + x;
    float t0 = p0[oy], t1 = p1[oy], t2 = p2[o];
    uint32_t k[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t j = 0; j < rows; ++j) {
        const float a0 = t0, a1 = t1, a2 = t2;
        if (j + 1 < rows) {
            const uint32_t on2 = yrow(y_lo + j + 1) * lx + x;
            t0 = p0[on2];
            t1 = p1[on2];
            t2 = p2[oy];
            oy = on2;
        }
        const float2 ry = proj2(a0, a1);
        float sn, cn;
        __sincosf(a2, &sn, &cn);
        const float2 rz = make_float2(r.y, wolff_projection(cn, sn, cphi, sphi));
        float2 rx = make_float2(__shfl_down_sync(0xffffffffu, r.x, 1), __shfl_down_sync(0xffffffffu, r.y, 1));
        const float ex = __shfl_sync(0xffffffffu, r_next.x, j), ey = __shfl_sync(0xffffffffu, r_next.y, j);
        if (lane + 1 == nv) rx = make_float2(ex, ey);
        const slsf_u32x4 b0 = slsf_stream(seed, counter, SLSF_PURPOSE_WOLFF_BOND, 0, z * plane + o);
        const slsf_u32x4 b1 = slsf_stream(seed, counter, SLSF_PURPOSE_WOLFF_BOND, 0, z1 * plane + o);
        const float2 jr = __fmul2_rn(jx, r);
        uint32_t v[6];
        wolff_bond_words(__fmul2_rn(jr, rx), m2b2, b0.x, b1.x, v[0], v[3]);
        wolff_bond_words(__fmul2_rn(jr, ry), m2b2, b0.y, b1.y, v[1], v[4]);
        wolff_bond_words(__fmul2_rn(__fmul2_rn(jzz, r), rz), m2b2, b0.z, b1.z, v[2], v[5]);
#pragma unroll
        for (int q = 0; q < 6; ++q) k[q] = lane == j ? v[q] : k[q];
        if (bond_bytes && lane < nv) {
            auto bits = [&](int q) {
                return (uint8_t)((v[q] >> lane & 1u) | (v[q + 1] >> lane & 1u) << 1 | (v[q + 2] >> lane & 1u) << 2);
            };
            bond_bytes[(size_t)z * plane + o] = bits(0);
            if (pair) bond_bytes[(size_t)z1 * plane + o] = bits(3);
        }
        r = ry;
        o += lx;
    }
    if (lane < rows) {
        const uint32_t m = 0xffffffffu >> (32u - nv);
        const uint32_t i = w + words * (y_lo + lane + ly * z), i1 = i + words * ly;
        wb.bx[i] = k[0] & m;
        wb.by[i] = k[1] & m;
        wb.bz[i] = k[2] & m;
        wb.cl[i] = 0u;
        if (pair) {
            wb.bx[i1] = k[3] & m;
            wb.by[i1] = k[4] & m;
            wb.bz[i1] = k[5] & m;
            wb.cl[i1] = 0u;
        }
    }
}

struct GrowGeo {
    uint32_t lx, ly, lz, words, ry_n, rz_n;
    bool px, py, pz; /* the region spans the whole period along x (one-word rows), y (32 rows), z (32 planes) */
};

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

__global__ void __launch_bounds__(kGrowThreads, 1)
    k_wb_grow(WolffBits wb, GrowGeo g, uint32_t max_items, unsigned long long* __restrict__ stats) {
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

/* Reflect the cluster's sites, count them; optional byte mask.  A thread
 * takes up to four consecutive sites of a row (one 16-byte access when L_x is
 * a multiple of 4 and the angles are aligned). */
__global__ void __launch_bounds__(kFlipThreads)
    k_wb_flip(float* __restrict__ theta, uint32_t lx, uint32_t rows, slsf_fastdiv quads, const uint32_t* __restrict__ cl,
              float phi, unsigned long long* __restrict__ stats, uint8_t* __restrict__ cluster_out, bool wide) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t n = 0;
    if (q < quads.d * rows) {
        const uint32_t row = slsf_fastdiv_div(q, quads), x = 4u * (q - row * quads.d), sites = min(4u, lx - x);
        const uint32_t m = (__ldcg(&cl[row * ((lx + 31u) >> 5) + (x >> 5)]) >> (x & 31u)) & 0xfu;
        const size_t i = (size_t)row * lx + x;
        if (m && wide) {
            float4 v = *reinterpret_cast<float4*>(theta + i);
            if (m & 1u) v.x = slsf_reflect(v.x, phi);
            if (m & 2u) v.y = slsf_reflect(v.y, phi);
            if (m & 4u) v.z = slsf_reflect(v.z, phi);
            if (m & 8u) v.w = slsf_reflect(v.w, phi);
            *reinterpret_cast<float4*>(theta + i) = v;
        } else if (m) {
            for (uint32_t k = 0; k < sites; ++k)
                if (m >> k & 1u) theta[i + k] = slsf_reflect(theta[i + k], phi);
        }
        n = __popc(m);
        if (cluster_out)
            for (uint32_t k = 0; k < sites; ++k) cluster_out[i + k] = (uint8_t)(m >> k & 1u);
    }
    __shared__ unsigned int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) n += __shfl_down_sync(0xffffffffu, n, off);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&s_sum, n);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(&stats[kStatClusterSites], (unsigned long long)s_sum);
}

uint32_t pow2_at_least(uint32_t n) {
    uint32_t p = 1;
    while (p < n) p <<= 1;
    return p;
}

}  // namespace

namespace {

uint64_t bit_words(uint32_t lx, uint32_t ly, uint32_t lz) { return (uint64_t)((lx + 31) / 32) * ly * lz; }

uint64_t bit_regions(uint32_t lx, uint32_t ly, uint32_t lz) {
    return (uint64_t)((lx + 31) / 32) * ((ly + kRegion - 1) / kRegion) * ((lz + kRegion - 1) / kRegion);
}

}  // namespace

uint64_t wolff_bits_scratch_bytes(uint32_t lx, uint32_t ly, uint32_t lz) {
    const uint64_t regions = bit_regions(lx, ly, lz);
    const uint64_t cap = pow2_at_least((uint32_t)std::min<uint64_t>(2 * regions + 2, 1u << 31));
    return 4 * round256(4 * bit_words(lx, ly, lz)) + round256(4 * regions) + round256(4 * cap) + 256;
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
    const uint64_t words = bit_words(t.lx, t.ly, t.lz);
    WolffBits wb;
    unsigned char* p = static_cast<unsigned char*>(scratch);
    wb.bx = reinterpret_cast<uint32_t*>(p);
    p += round256(4 * words);
    wb.by = reinterpret_cast<uint32_t*>(p);
    p += round256(4 * words);
    wb.bz = reinterpret_cast<uint32_t*>(p);
    p += round256(4 * words);
    wb.cl = reinterpret_cast<uint32_t*>(p);
    p += round256(4 * words);
    wb.regions = (uint32_t)bit_regions(t.lx, t.ly, t.lz);
    wb.cap = pow2_at_least(2 * wb.regions + 2);
    unsigned char* control = p;
    wb.queued = reinterpret_cast<uint32_t*>(p);
    p += round256(4ull * wb.regions);
    wb.ring = reinterpret_cast<uint32_t*>(p);
    p += round256(4ull * wb.cap);
    wb.ctl = reinterpret_cast<uint32_t*>(p);
    p += 256;
    cudaMemsetAsync(control, 0, (size_t)(p - control), s);
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
    GrowGeo g;
    g.lx = t.lx;
    g.ly = t.ly;
    g.lz = t.lz;
    g.words = (t.lx + 31) / 32;
    g.ry_n = (t.ly + kRegion - 1) / kRegion;
    g.rz_n = (t.lz + kRegion - 1) / kRegion;
    g.px = g.words == 1;
    g.py = t.ly == kRegion;
    g.pz = t.lz == kRegion;
    const uint32_t grid = std::min<uint32_t>(wb.regions, (uint32_t)sms);
    /* every region is processed at most once per bit it gains */
    const uint32_t max_items = t.loop_limit ? t.loop_limit : std::max<uint32_t>(64, volume / 32);
    k_wb_grow<<<grid, kGrowThreads, 0, s>>>(wb, g, max_items, t.stats);
    const slsf_fastdiv quads = slsf_fastdiv_make((t.lx + 3) / 4);
    const uint32_t rows = t.ly * t.lz;
    const bool wide = t.lx % 4 == 0 && (reinterpret_cast<uintptr_t>(t.theta) & 15u) == 0;
    k_wb_flip<<<(quads.d * rows + kFlipThreads - 1) / kFlipThreads, kFlipThreads, 0, s>>>(
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
