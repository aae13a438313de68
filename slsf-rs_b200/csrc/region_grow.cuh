/*
 * Growth of a Wolff cluster on bit-packed bonds by regions, for
 * kernel_wolff_bits.cu (one lattice per launch) and kernel_stream.cu (several
 * CTAs of a replica when there are few replicas).
 *
 * The lattice is cut into regions of one word (32 sites along x) by 32 rows by
 * 32 planes; a word past a row's end and rows and planes past the lattice hold
 * zeros.  A CTA takes a region from a work queue, reads its cluster and bond
 * words into shared memory with the bits that enter through the region's faces,
 * closes it (bitgrow.cuh), ORs the result back and queues every neighbour
 * region its bits can enter.  CTAs only wait for work that running CTAs hold,
 * so no co-residency is needed.  Bits only ever get set, so the fixed point is
 * the seed's component whatever the order.  Every wait and loop is bounded;
 * past a bound kErrGrowthLimit goes to the task's error word.
 */
#ifndef SLSF_REGION_GROW_CUH
#define SLSF_REGION_GROW_CUH

#include "bitgrow.cuh"
#include "engine.h"

namespace slsf {

constexpr uint32_t kRegion = kGrowEdge; /* region edge in sites along y and z; one word along x */
constexpr uint32_t kGrowThreads = kRegion * kRegion;
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
template <int kT>
__device__ __forceinline__ bool grow_region(const WolffBits& wb, const GrowGeo& g, uint32_t r, uint32_t seed_word, uint32_t seed_bit,
                            uint32_t (*C)[kRegion + 1], uint32_t (*BY)[kRegion + 1], uint32_t (*BZ)[kRegion + 1],
                            uint32_t (*BX)[kRegion + 1], uint32_t* keep, uint32_t* s_want) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t k = r % g.words, rest = r / g.words, ry = rest % g.ry_n, rz = rest / g.ry_n;
    const uint32_t rowlen = g.words; /* words per row */
    /* the thread's words: row `lane` of the planes warp, warp + 32 / kT, ... */
    const uint32_t gy = ry * kRegion + lane;
    const bool last_y = lane == kRegion - 1 || gy + 1 == g.ly;
    auto plane_of = [&](int p) { return warp + p * (kRegion / kT); };
    /* rows and planes past the lattice hold zeros; the last ones of a region face the next region */
    auto inside = [&](int p) { return gy < g.ly && rz * kRegion + plane_of(p) < g.lz; };
    auto last_z = [&](int p) { return plane_of(p) == kRegion - 1 || rz * kRegion + plane_of(p) + 1 == g.lz; };
    /* the word's last site, and that of the word to its left */
    const uint32_t top = min(32u, g.lx - 32u * k) - 1, kl = k == 0 ? g.words - 1 : k - 1;
    const uint32_t top_l = min(32u, g.lx - 32u * kl) - 1;
    auto word = [&](uint32_t kk, uint32_t yy, uint32_t zz) { return kk + rowlen * (yy + g.ly * zz); };
#ifdef SLSF_WB_STATS
    long long tclk = clock64();
#endif
    /* the region's own words (written only by processings of this region) */
    uint32_t w[kT], c0[kT], c[kT], bxw[kT], byw[kT], bzw[kT], bxi[kT];
#pragma unroll
    for (int p = 0; p < kT; ++p) {
        const bool in = inside(p);
        w[p] = in ? word(k, gy, rz * kRegion + plane_of(p)) : 0u;
        c[p] = c0[p] = in ? __ldcg(&wb.cl[w[p]]) : 0u;
        bxw[p] = in ? wb.bx[w[p]] : 0u;
        byw[p] = in ? wb.by[w[p]] : 0u;
        bzw[p] = in ? wb.bz[w[p]] : 0u;
    }
    /* claimable again from here on: the reset is visible before the
     * neighbours' words are read, so a neighbour that adds face bits later
     * finds the region unqueued and queues it */
    if (threadIdx.x == 0) {
        wb.queued[r] = 0u;
        __threadfence();
    }
    __syncthreads();
    /* bits entering through the faces.  The faces' neighbour words as loaded
     * here also decide, at the end, which neighbours to queue: a neighbour
     * word only ever gains bits, so a stale copy can queue a region that needs
     * nothing, never miss one.  out_*: bits that the neighbour takes and does not have. */
    const uint32_t kr = k + 1 == g.words ? 0 : k + 1;
    const uint32_t ym = gy == 0 ? g.ly - 1 : gy - 1, yp = gy + 1 == g.ly ? 0 : gy + 1;
    uint32_t out_x[kT], out_ym[kT], out_yp[kT], out_zm[kT], out_zp[kT]; /* out_x: bit 0 to the left, bit 1 to the right */
    int fresh = 0;
#pragma unroll
    for (int p = 0; p < kT; ++p) {
        const bool in = inside(p);
        const uint32_t gz = rz * kRegion + plane_of(p);
        out_x[p] = out_ym[p] = out_yp[p] = out_zm[p] = out_zp[p] = 0;
        if (!g.px && in) {
            const uint32_t wl = word(kl, gy, gz), wr = word(kr, gy, gz);
            const uint32_t cl_l = __ldcg(&wb.cl[wl]) >> top_l & 1u, bx_l = wb.bx[wl] >> top_l & 1u, cl_r = __ldcg(&wb.cl[wr]) & 1u;
            c[p] |= cl_l & bx_l;
            c[p] |= (cl_r & (bxw[p] >> top)) << top;
            out_x[p] = (bx_l & ~cl_l) | (bxw[p] >> top & ~cl_r & 1u) << 1;
        }
        if (!g.py && in) {
            if (lane == 0) {
                const uint32_t wm = word(k, ym, gz), cl_ym = __ldcg(&wb.cl[wm]), by_ym = wb.by[wm];
                c[p] |= cl_ym & by_ym;
                out_ym[p] = by_ym & ~cl_ym;
            }
            if (last_y) {
                const uint32_t cl_yp = __ldcg(&wb.cl[word(k, yp, gz)]);
                c[p] |= cl_yp & byw[p];
                out_yp[p] = byw[p] & ~cl_yp;
            }
        }
        if (!g.pz && in) {
            if (plane_of(p) == 0) {
                const uint32_t wm = word(k, gy, gz == 0 ? g.lz - 1 : gz - 1), cl_zm = __ldcg(&wb.cl[wm]), bz_zm = wb.bz[wm];
                c[p] |= cl_zm & bz_zm;
                out_zm[p] = bz_zm & ~cl_zm;
            }
            if (last_z(p)) {
                const uint32_t cl_zp = __ldcg(&wb.cl[word(k, gy, gz + 1 == g.lz ? 0 : gz + 1)]);
                c[p] |= cl_zp & bzw[p];
                out_zp[p] = bzw[p] & ~cl_zp;
            }
        }
        if (in && seed_word == w[p]) c[p] |= 1u << seed_bit;
        /* inside the word: bond bit `top` of an open word leads out of it */
        bxi[p] = g.px ? bxw[p] : bxw[p] & ((1u << top) - 1u);
        c[p] = g.px ? close_word(c[p], bxi[p], g.lx, true) : close_word(c[p], bxi[p], 32u, false);
        fresh |= c[p] != c0[p];
    }
    /* the stored region is closed already: without new bits nothing changes */
    const int any_new = __syncthreads_or(fresh);
    SLSF_WB_CLOCK(5, tclk);
    if (!any_new) {
        SLSF_WB_COUNT(3, 1);
        return true;
    }
#pragma unroll
    for (int p = 0; p < kT; ++p) {
        const uint32_t z = plane_of(p);
        C[z][lane] = c[p];
        BX[z][lane] = bxi[p];
        BY[z][lane] = last_y && !g.py ? 0u : byw[p]; /* the bonds out of the region are the faces' */
        BZ[z][lane] = last_z(p) && !g.pz ? 0u : bzw[p];
    }
    __syncthreads();
    const GrowBlock q = {&C[0][0], &BX[0][0], &BY[0][0], &BZ[0][0], g.px ? g.lx : 32u, g.px, g.py, g.pz};
    const uint32_t passes = close_block<kT>(q, kRegion * kRegion * kRegion + 1);
    SLSF_WB_COUNT(1, passes);
    SLSF_WB_CLOCK(6, tclk);
    const bool ok = passes != 0;
    /* neighbours that the region's bits can enter: bit 0/1 -x/+x, 2/3 -y/+y, 4/5 -z/+z */
    uint32_t want = 0;
#pragma unroll
    for (int p = 0; p < kT; ++p) {
        const uint32_t v = C[plane_of(p)][lane];
        if (inside(p) && v != c0[p]) atomicOr(&wb.cl[w[p]], v);
        if (v & out_x[p] & 1u) want |= 1u;
        if ((v >> top) & (out_x[p] >> 1) & 1u) want |= 2u;
        if (v & out_ym[p]) want |= 4u;
        if (v & out_yp[p]) want |= 8u;
        if (v & out_zm[p]) want |= 16u;
        if (v & out_zp[p]) want |= 32u;
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

/* Takes regions until nothing is queued or in flight (1024 / kT threads). */
template <int kT>
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
        ok &= grow_region<kT>(wb, g, r, seed_word, seed_bit, C, BY, BZ, BX, &s_keep, &s_want);
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

}  // namespace slsf

#endif /* SLSF_REGION_GROW_CUH */
