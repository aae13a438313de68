/*
 * Many replicas too large for one CTA's shared memory, their state in global
 * memory (L2 holds about a hundred 64^3 lattices): the sweeps, Wolff updates
 * and measurements of all of them in one persistent launch.  Same role as
 * kernel_resident.cu -- the carlo-mc Runner's task-by-task loop over
 * ThetaModel::sweep + ThetaModel::measure (src/model.rs:379-442,
 * src/results.rs:200-202) -- for rows of up to 64 sites, L_x a multiple of 4.
 *
 * A replica's sweep is a sequence of phases -- colour 0 (with the measurement
 * of the state it starts from), colour 1, and per Wolff step bond activation,
 * growth and reflection -- each cut into chunks of one CTA's work (growth is
 * one chunk).  CTAs take chunks from a queue in order; the CTA that finishes a
 * phase's last chunk queues the next phase of that replica.  So replicas
 * advance independently of each other: the growth of one (a latency-bound
 * chain, 65 to 200 us at 64^3 depending on the cluster) runs beside the sweeps
 * of the others, which a launch per phase for all replicas cannot do (every
 * phase would wait for its slowest growth: 300 us per sweep of 32 replicas
 * against 83 us of other work).  CTAs wait only for chunks that running CTAs
 * will queue, so no co-residency is needed; every wait is bounded.
 *
 * Visibility: a chunk's writes are fenced before its replica's counter is
 * decremented, the next phase's entries are written after the counter reached
 * zero, and a CTA fences after it has read its entry, before it reads the
 * replica.
 */
#include <algorithm>
#include <type_traits>

#include "engine.h"
#include "region_grow.cuh"
#include "walk_global.cuh"
#include "wolff_global.cuh"

namespace slsf {

namespace {

constexpr uint32_t kStreamThreads = 512; /* one CTA per SM: 128 registers a thread */
constexpr uint32_t kStreamRows = 8;      /* rows per thread in the growth */
constexpr uint32_t kFlipQuads = 8;       /* quads per thread of a reflection */
constexpr uint32_t kRingEntries = 1u << 20;
constexpr uint32_t kChunkBits = 12;
constexpr uint32_t kMaxWolffSteps = 1024;

enum Phase : uint32_t { kColour0, kColour1, kBonds, kGrow, kFlip, kMeasureLast, kDone };

/* One replica's place in the launch. */
struct StreamCtl {
    uint32_t left; /* chunks of the phase not yet finished */
    uint32_t phase, sweep, step;
};

/* Sizes of the chunks of a launch.  A phase is a row of blocks of one CTA's
 * threads (walks of walk_planes planes per thread, a run of rows per warp,
 * kFlipQuads quads per thread); a chunk takes `per` of them one after the other.  The
 * blocks, and so the order of the measured sums, are the same in every launch. */
struct StreamShape {
    uint32_t per;      /* blocks per chunk */
    uint32_t bond_run; /* rows per warp of the bond activation */
    uint32_t planes;   /* planes per thread of colour 1, at most; 0: as colour 0 */
    uint32_t growers;  /* CTAs that grow a replica's cluster together by regions; 1: one CTA by rows */
};

__host__ __device__ inline uint32_t smaller(uint32_t a, uint32_t b) { return a < b ? a : b; }

/* Planes per thread of a replica's walks, for colour 0 and the measurement by its
 * size alone: the order of the measured sums hangs on it.  Fewer planes shorten a
 * lone replica's phases and start more walks (us per sweep, 4 and 8 planes: one 40^3 84 / 96, one 56^3 109
 * / 120, thirty-two 64x64x40 137 / 144); the largest replicas fill the GPU with
 * 8 already (thirty-two 64^3 233 / 218). */
__host__ __device__ inline uint32_t walk_planes(const TaskView& t, const StreamShape& sh, uint32_t phase) {
    if (phase == kColour1 && sh.planes) return sh.planes;
    return t.lx * t.ly * t.lz >= 200000 ? 8 : 4;
}

__host__ __device__ inline uint32_t blocks_of(const TaskView& t, const StreamShape& sh, uint32_t phase) {
    switch (phase) {
        case kColour0:
        case kColour1:
        case kMeasureLast: return (walk_units(t, walk_planes(t, sh, phase)) + kStreamThreads - 1) / kStreamThreads;
        case kBonds: {
            const uint32_t warps = ((t.lx + 31) / 32) * (t.lz / 2) * ((t.ly + sh.bond_run - 1) / sh.bond_run);
            return (warps + kStreamThreads / 32 - 1) / (kStreamThreads / 32);
        }
        case kFlip: return ((t.lx >> 2) * t.ly * t.lz + kStreamThreads * kFlipQuads - 1) / (kStreamThreads * kFlipQuads);
        default: return 0;
    }
}

__host__ __device__ inline uint32_t chunks_of(const TaskView& t, const StreamShape& sh, uint32_t phase) {
    if (phase == kGrow) return smaller(sh.growers, (uint32_t)bit_regions(t.lx, t.ly, t.lz));
    return (blocks_of(t, sh, phase) + sh.per - 1) / sh.per;
}

/* The phase after `c` for sweeps below sw_hi of the launch. */
__device__ __forceinline__ StreamCtl next_phase(const TaskView& t, const StreamShape& sh, StreamCtl c, uint32_t sw_hi) {
    bool sweep_done = false;
    switch (c.phase) {
        case kColour0: c.phase = kColour1; break;
        case kColour1:
            c.step = 0;
            if (t.wolff_steps) c.phase = kBonds;
            else sweep_done = true;
            break;
        case kBonds: c.phase = kGrow; break;
        case kGrow: c.phase = kFlip; break;
        case kFlip:
            if (++c.step < t.wolff_steps) c.phase = kBonds;
            else sweep_done = true;
            break;
        default: c.phase = kDone; break;
    }
    if (sweep_done) {
        ++c.sweep;
        if (c.sweep < min(t.sweeps, sw_hi)) c.phase = kColour0;
        else c.phase = c.sweep == t.sweeps && t.n_bins ? kMeasureLast : kDone;
    }
    c.left = chunks_of(t, sh, c.phase);
    return c;
}

struct StreamQueue {
    unsigned long long* ring; /* entry of ticket q: (q + 1) << 32 | replica << kChunkBits | chunk */
    uint32_t* head;           /* tickets taken */
    uint32_t* tail;           /* entries queued */
    uint32_t* abort;          /* a wait ran out */
};

__device__ __forceinline__ void put_entry(const StreamQueue& q, uint32_t at, uint32_t replica, uint32_t chunk) {
    *(volatile unsigned long long*)&q.ring[at] = (unsigned long long)(at + 1) << 32 | replica << kChunkBits | chunk;
}

__device__ __forceinline__ BitPlanes stream_planes(const TaskView& t) {
    const WolffBits wb = carve_bits(t.bits, t.lx, t.ly, t.lz);
    return {wb.bx, wb.by, wb.bz, wb.cl};
}

/* Growth of a replica's cluster by the CTA, row words W of up to 32 or 64
 * sites: row passes as in the one-CTA kernel (kernel_resident.cu), R rows per
 * thread with their bonds in registers, the cluster words in shared memory,
 * three steps per block barrier.  At 64^3 about 49 steps of 2,500 cycles, bound
 * by instruction issue (visits of marked rows only, closures of whole lines by
 * segments and scans by shuffles were no faster: 129k, 140k and more cycles
 * against 122k). */
template <typename W, int R, bool kWhole>
__device__ __forceinline__ bool grow_replica(const TaskView& t, const slsf_u32x4& pick, volatile W* cl) {
    const uint32_t lx = t.lx, ly = t.ly, lz = t.lz, rows = ly * lz;
    const BitPlanes planes = stream_planes(t);
    const W *bx = reinterpret_cast<const W*>(planes.bx), *by = reinterpret_cast<const W*>(planes.by),
            *bz = reinterpret_cast<const W*>(planes.bz);
    const uint32_t seed_row = slsf_range(pick.z, ly) + ly * slsf_range(pick.w, lz);
    W b_yp[R], b_ym[R], b_zp[R], b_zm[R], b_x[R];
    uint32_t y_nb[R], z_nb[R]; /* the neighbouring rows: below in the low half, above in the high half */
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const uint32_t r = threadIdx.x + j * kStreamThreads;
        b_yp[j] = b_ym[j] = b_zp[j] = b_zm[j] = b_x[j] = 0;
        y_nb[j] = z_nb[j] = 0;
        if (r < rows) {
            const uint32_t z = r / ly, y = r - z * ly;
            const uint32_t ym = y == 0 ? r + ly - 1 : r - 1, yp = y + 1 == ly ? r + 1 - ly : r + 1;
            const uint32_t zm = z == 0 ? r + rows - ly : r - ly, zp = z + 1 == lz ? r + ly - rows : r + ly;
            b_yp[j] = by[r];
            b_ym[j] = by[ym];
            b_zp[j] = bz[r];
            b_zm[j] = bz[zm];
            b_x[j] = bx[r];
            y_nb[j] = ym | yp << 16;
            z_nb[j] = zm | zp << 16;
            cl[r] = r == seed_row ? close_row<kWhole>((W)1 << slsf_range(pick.y, lx), b_x[j], lx) : (W)0;
        }
    }
    __syncthreads();
    constexpr int kSteps = 3;
    const uint32_t bound = (t.loop_limit ? min(t.loop_limit, lx * rows) : lx * rows) + 1;
    bool closed = false;
    for (uint32_t pass = 0; pass < bound && !closed; ++pass) {
        int changed = 0;
#pragma unroll 1
        for (int step = 0; step < kSteps; ++step) {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint32_t r = threadIdx.x + j * kStreamThreads;
                if (r < rows) {
                    const W in = (cl[y_nb[j] & 0xffffu] & b_ym[j]) | (cl[y_nb[j] >> 16] & b_yp[j]) |
                                 (cl[z_nb[j] & 0xffffu] & b_zm[j]) | (cl[z_nb[j] >> 16] & b_zp[j]);
                    const W old = cl[r], c = old | in;
                    if (c != old) {
                        cl[r] = close_row<kWhole>(c, b_x[j], lx);
                        changed = 1;
                    }
                }
            }
        }
        closed = !__syncthreads_or(changed);
    }
    W* out = reinterpret_cast<W*>(planes.cl);
    for (uint32_t r = threadIdx.x; r < rows; r += kStreamThreads) out[r] = cl[r];
    return closed;
}

/* Adds a per-thread count to stats[slot]. */
__device__ __forceinline__ void count_into(uint32_t v, unsigned long long* stats, int slot) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&stats[slot], (unsigned long long)v);
}

__global__ void k_stream_init(const TaskView* __restrict__ views, StreamCtl* __restrict__ ctl, StreamQueue q, uint32_t n,
                              StreamShape sh, uint32_t sw_lo, uint32_t sw_hi) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const TaskView t = views[i];
    if (sw_lo >= min(t.sweeps, sw_hi)) return;
    const StreamCtl c = {chunks_of(t, sh, kColour0), kColour0, sw_lo, 0};
    ctl[i] = c;
    const uint32_t at = atomicAdd(q.tail, c.left);
    for (uint32_t k = 0; k < c.left; ++k) put_entry(q, at + k, i, k);
}

__global__ void __launch_bounds__(kStreamThreads, 1)
    k_stream(const TaskView* __restrict__ views, const unsigned long long* __restrict__ counters, StreamCtl* ctl,
             StreamQueue q, uint32_t tickets, StreamShape sh, uint32_t sw_hi) {
    extern __shared__ __align__(8) unsigned char grow_smem[]; /* the growth's cluster words */
    __shared__ double scratch[8 * 32];
    __shared__ uint32_t s_entry, s_at;
    __shared__ StreamCtl s_ctl;
    __shared__ bool s_last;
    constexpr uint32_t kNone = 0xffffffffu, kSpin = 1u << 26;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t got = kNone;
            const uint32_t ticket = atomicAdd(q.head, 1u);
            if (ticket < tickets) {
                volatile unsigned long long* e = q.ring + ticket;
                for (uint32_t spin = 0;; ++spin) {
                    const unsigned long long v = *e;
                    if ((uint32_t)(v >> 32) == ticket + 1) {
                        got = (uint32_t)v;
                        break;
                    }
                    if (*(volatile uint32_t*)q.abort) break;
                    if (spin == kSpin) {
                        atomicOr(&views[0].stats[kStatError], kErrQueueLimit);
                        atomicExch(q.abort, 1u);
                        break;
                    }
                    __nanosleep(64);
                }
                __threadfence();
                if (got != kNone) {
                    const uint4 c = __ldcg(reinterpret_cast<const uint4*>(&ctl[got >> kChunkBits]));
                    s_ctl = {c.x, c.y, c.z, c.w};
                }
            }
            s_entry = got;
        }
        __syncthreads();
        if (s_entry == kNone) return;
        const uint32_t replica = s_entry >> kChunkBits, chunk = s_entry & ((1u << kChunkBits) - 1);
        const StreamCtl c = s_ctl;
        const TaskView t = views[replica];
        const uint64_t sweep = (counters ? counters[2 * replica] : t.metro_sweeps) + c.sweep;
        const uint64_t counter = (counters ? counters[2 * replica + 1] : t.wolff_done) + (uint64_t)c.sweep * t.wolff_steps + c.step;
        /* bin row of the state that colour 0 starts from, or of the last state */
        double* bin_row = nullptr;
        if ((c.phase == kColour0 && c.sweep > 0) || c.phase == kMeasureLast) bin_row = bin_row_of(t, sweep);
        const uint32_t planes = walk_planes(t, sh, c.phase);
        const uint32_t b_lo = chunk * sh.per, b_hi = smaller(b_lo + sh.per, blocks_of(t, sh, c.phase));
        if (c.phase == kColour1 || (c.phase == kColour0 && !bin_row)) {
            uint32_t accepted = 0;
            for (uint32_t b = b_lo; b < b_hi; ++b)
                accepted += walk_colour<false>(t, sweep, c.phase == kColour1, planes, b * kStreamThreads + threadIdx.x, nullptr);
            count_into(accepted, t.stats, kStatAccepted);
        } else if (c.phase == kColour0 || c.phase == kMeasureLast) {
            uint32_t accepted = 0;
            for (uint32_t b = b_lo; b < b_hi && bin_row; ++b) {
                WalkSums sums;
                sums.start(t.jxy_max, t.jz_max);
                const uint32_t unit = b * kStreamThreads + threadIdx.x;
                if (c.phase == kColour0)
                    accepted += walk_colour<true>(t, sweep, 0, planes, unit, &sums);
                else
                    walk_measure(t, planes, unit, sums);
                block_sum<8>(sums.acc, scratch);
                if (threadIdx.x == 0)
#pragma unroll
                    for (int k = 0; k < 8; ++k) t.partials[b * 8 + k] = sums.acc[k];
            }
            if (c.phase == kColour0) count_into(accepted, t.stats, kStatAccepted);
        } else {
            const slsf_u32x4 pick = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_PICK, 0, 0);
            const float phi = slsf_angle_from_word(pick.x);
            if (c.phase == kBonds) {
                if (chunk == 0 && sh.growers > 1) { /* the region queue, with the seed's region its first entry */
                    const WolffBits wb = carve_bits(t.bits, t.lx, t.ly, t.lz);
                    const uint32_t n = (uint32_t)(control_bytes(wb.regions) / 4);
                    for (uint32_t i = threadIdx.x; i < n; i += kStreamThreads) wb.queued[i] = 0;
                    __syncthreads();
                    if (threadIdx.x == 0)
                        queue_seed(wb, t.lx, t.ly, t.lz, slsf_range(pick.y, t.lx), slsf_range(pick.z, t.ly),
                                   slsf_range(pick.w, t.lz));
                }
                const BitPlanes planes = stream_planes(t);
                for (uint32_t b = b_lo; b < b_hi; ++b)
                    bond_run<2>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, __fmul_rn(-2.0f, t.beta), phi, t.seed, counter, planes,
                                sh.bond_run, (b * kStreamThreads + threadIdx.x) >> 5, nullptr);
            } else if (c.phase == kGrow && sh.growers > 1) {
                grow_regions<2>(carve_bits(t.bits, t.lx, t.ly, t.lz), grow_geo(t.lx, t.ly, t.lz),
                                t.loop_limit ? t.loop_limit : max(64u, t.lx * t.ly * t.lz / 32), t.stats);
                if (chunk == 0 && threadIdx.x == 0) atomicAdd(&t.stats[kStatClusters], 1ull);
            } else if (c.phase == kGrow) {
                uint32_t* cl = reinterpret_cast<uint32_t*>(grow_smem);
                uint64_t* cl2 = reinterpret_cast<uint64_t*>(grow_smem);
                const bool closed = t.lx <= 32 ? grow_replica<uint32_t, kStreamRows, false>(t, pick, cl)
                                    : t.lx == 64 ? grow_replica<uint64_t, kStreamRows, true>(t, pick, cl2)
                                                 : grow_replica<uint64_t, kStreamRows, false>(t, pick, cl2);
                if (threadIdx.x == 0) {
                    if (!closed) atomicOr(&t.stats[kStatError], kErrGrowthLimit);
                    atomicAdd(&t.stats[kStatClusters], 1ull);
                }
            } else {
                const slsf_fastdiv quads = slsf_fastdiv_make(t.lx >> 2);
                const uint32_t* cl = stream_planes(t).cl;
                uint32_t members = 0;
                for (uint32_t j = b_lo * kFlipQuads; j < b_hi * kFlipQuads; j += 4)
                    members += flip_quads<4>(t.theta, t.lx, t.ly * t.lz, j * kStreamThreads + threadIdx.x, kStreamThreads, quads,
                                             cl, phi, nullptr, true);
                count_into(members, t.stats, kStatClusterSites);
            }
        }
        /* the chunk's writes, then its count; the last chunk of the phase queues the next phase */
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicSub(&ctl[replica].left, 1u) == 1u;
            if (s_last) __threadfence();
        }
        __syncthreads();
        if (!s_last) continue;
        if (bin_row) { /* the blocks' sums in order */
            if (threadIdx.x < 8) {
                double a = 0.0;
                for (uint32_t k = 0; k < blocks_of(t, sh, c.phase); ++k) a += __ldcg(&t.partials[k * 8 + threadIdx.x]);
                scratch[threadIdx.x] = a;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const double tot[8] = {scratch[0], scratch[1], scratch[2], scratch[3],
                                       scratch[4], scratch[5], scratch[6], scratch[7]};
                add_to_bin(t, tot, bin_row);
            }
        }
        const StreamCtl nx = next_phase(t, sh, c, sw_hi);
        if (nx.phase == kDone) continue;
        if (threadIdx.x == 0) {
            __stcg(reinterpret_cast<uint4*>(&ctl[replica]), make_uint4(nx.left, nx.phase, nx.sweep, nx.step));
            __threadfence();
            s_at = atomicAdd(q.tail, nx.left);
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < nx.left; k += kStreamThreads) {
            __threadfence();
            put_entry(q, s_at + k, replica, k);
        }
    }
}

/* Advances the counters of a replayed launch. */
__global__ void k_stream_advance(const TaskView* __restrict__ views, unsigned long long* __restrict__ counters, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    counters[2 * i] += views[i].sweeps;
    counters[2 * i + 1] += (uint64_t)views[i].sweeps * views[i].wolff_steps;
}

uint64_t items_per_sweep(const TaskView& t, const StreamShape& sh) {
    return (uint64_t)chunks_of(t, sh, kColour0) + chunks_of(t, sh, kColour1) +
           (uint64_t)t.wolff_steps * (chunks_of(t, sh, kBonds) + chunks_of(t, sh, kGrow) + chunks_of(t, sh, kFlip));
}

}  // namespace

bool stream_fits(uint32_t lx, uint32_t ly, uint32_t lz) {
    /* patches of four sites by two rows, plane pairs, one or two words per row, the growth's rows and 16-bit row numbers;
     * the chunk numbers; the bit planes in 4 V bytes */
    return lx >= 4 && lx <= 64 && lx % 4 == 0 && ly >= 2 && ly % 2 == 0 && lz >= 2 && lz % 2 == 0 &&
           (uint64_t)ly * lz <= (uint64_t)kStreamThreads * kStreamRows &&
           wolff_bits_scratch_bytes(lx, ly, lz) <= 4ull * lx * ly * lz;
}

bool stream_takes(const TaskView& t) { return walk_supports(t) && t.wolff_steps <= kMaxWolffSteps; }

size_t stream_scratch_bytes(uint32_t n) { return 256 + sizeof(StreamCtl) * (size_t)n + 8ull * kRingEntries; }

cudaError_t launch_stream(const TaskView* views, const TaskView* host_views, unsigned long long* counters, uint32_t n, int sms,
                          void* scratch, cudaStream_t s, uint64_t* launches) {
    unsigned char* p = static_cast<unsigned char*>(scratch);
    StreamQueue q;
    q.head = reinterpret_cast<uint32_t*>(p);
    q.tail = q.head + 1;
    q.abort = q.head + 2;
    q.ring = reinterpret_cast<unsigned long long*>(p + 256);
    StreamCtl* ctl = reinterpret_cast<StreamCtl*>(p + 256 + 8ull * kRingEntries);
    /* as many blocks per chunk as leave three chunks of the walks per SM (each
     * chunk costs about 2 us in the queue and its fences: 1.42 against 1.28 ms per
     * sweep of 300 replicas of 64^3) */
    StreamShape sh = {8, 16, 0, 1};
    uint64_t sites = 0, gain = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const TaskView& t = host_views[i];
        const uint64_t chain = (t.lx + 31) / 32 + (t.ly + kRegion - 1) / kRegion + (t.lz + kRegion - 1) / kRegion;
        sites = std::max(sites, (uint64_t)t.lx * t.ly * t.lz);
        gain = std::max(gain, (uint64_t)t.ly * t.lz * (t.ly + t.lz) / (kStreamThreads * chain));
    }
    auto chunks = [&]() {
        uint64_t c = 0;
        for (uint32_t i = 0; i < n && c < 3ull * sms; ++i) c += chunks_of(host_views[i], sh, kColour0);
        return c;
    };
    while (sh.per > 1 && chunks() < 3ull * sms) sh.per >>= 1;
    /* Few walks: shorter phases, in colour 1's planes and the bonds' rows, which
     * no sum's order hangs on.  us per sweep with 16 rows, 8, 8 and two planes, 4 and
     * two planes: one 64x64x40 102 / 99 / 98 / 94, eight 116 / 113 / 111 / 107; one
     * 64^3 121 / 113 / 111 / 106, twelve 138 / 135 / 131 / 135; thirty-two 36x40x44
     * 103 / 101 / 98 / 104; sixteen 64x64x40, more walks than SMs, 121 / 119 / 120 / 125. */
    if (const uint64_t walks = chunks(); walks < (uint64_t)sms) {
        sh.planes = 2;
        sh.bond_run = 8 * walks < 5ull * sms ? 4 : 8;
    }
    /* Several CTAs grow a replica together, by regions, where one CTA's row
     * passes would take long and while there are SMs for them.  A pass visits
     * rows / 512 rows a thread and there are as many as the cluster is long,
     * L_y + L_z; the regions are a chain of their number along the axes: `gain` is
     * the one over the other.  us per sweep at T = 0.9, by rows / by 8 CTAs: one
     * 40^3 (gain 42) 85 / 90, 48^3 (72) 98 / 96, 36x4x512 (108) 189 / 157, 56^3
     * (114) 114 / 104, 36x256x12 (146) 215 / 121, 64^3 (170) 151 / 119, 36x8x512
     * (219) 276 / 176; sixteen 48^3 109 / 113, 56^3 137 / 126, 64^3 175 / 143,
     * 36x8x512 369 / 206.  Four CTAs each for up to 37 replicas pay at the larger
     * gains alone (thirty-two 56^3 145 / 171, 36x256x12 273 / 190, 64^3 248 / 236,
     * 36x8x512 375 / 310). */
    if (gain > 140)
        while (sh.growers < 8 && 2ull * sh.growers * n <= (uint64_t)sms) sh.growers <<= 1;
    else if ((gain > 100 || sites >= 150000) && 8ull * n <= (uint64_t)sms)
        sh.growers = 8;
    if (sh.growers < 4) sh.growers = 1;
    uint64_t most = 1;
    uint32_t rows = 0, sweeps = 0;
    for (uint32_t i = 0; i < n; ++i) {
        most = std::max(most, items_per_sweep(host_views[i], sh) + chunks_of(host_views[i], sh, kMeasureLast));
        rows = std::max(rows, host_views[i].ly * host_views[i].lz * (host_views[i].lx > 32 ? 2u : 1u));
        sweeps = std::max(sweeps, host_views[i].sweeps);
    }
    /* the largest growth's words, whatever this launch needs: another thread's launch may need more */
    cudaError_t e = cudaFuncSetAttribute(k_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(8 * kStreamThreads * kStreamRows));
    /* every launch's entries fit the ring: pieces of replicas, and of sweeps */
    const uint32_t piece = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(n, 1u << (32 - kChunkBits)), kRingEntries / most);
    for (uint32_t lo = 0; lo < n && e == cudaSuccess; lo += piece) {
        const uint32_t m = std::min(piece, n - lo);
        const TaskView* h = host_views + lo;
        unsigned long long* c = counters ? counters + 2 * lo : nullptr;
        const uint32_t span = (uint32_t)std::max<uint64_t>(1, kRingEntries / (most * m) > 1 ? kRingEntries / (most * m) - 1 : 1);
        for (uint32_t sw = 0; sw < sweeps && e == cudaSuccess; sw += span) {
            const uint32_t hi = std::min(sweeps, sw + span);
            uint64_t tickets = 0, wide = 0;
            for (uint32_t i = 0; i < m; ++i) {
                if (sw >= h[i].sweeps) continue;
                const uint32_t end = std::min(hi, h[i].sweeps);
                tickets += (end - sw) * items_per_sweep(h[i], sh);
                if (end == h[i].sweeps && h[i].n_bins) tickets += chunks_of(h[i], sh, kMeasureLast);
                wide += std::max(std::max(chunks_of(h[i], sh, kColour0), chunks_of(h[i], sh, kColour1)), chunks_of(h[i], sh, kBonds));
            }
            if (tickets == 0) continue;
            if (e == cudaSuccess) e = cudaMemsetAsync(scratch, 0, 256 + 8 * tickets, s);
            if (e != cudaSuccess) break;
            k_stream_init<<<(m + 127) / 128, 128, 0, s>>>(views + lo, ctl + lo, q, m, sh, sw, hi);
            k_stream<<<(uint32_t)std::min<uint64_t>(wide, (uint64_t)sms), kStreamThreads, 4 * rows, s>>>(
                views + lo, c, ctl + lo, q, (uint32_t)tickets, sh, hi);
            *launches += 2;
            e = cudaGetLastError();
        }
        if (c && e == cudaSuccess) {
            k_stream_advance<<<(m + 127) / 128, 128, 0, s>>>(views + lo, c, m);
            *launches += 1;
            e = cudaGetLastError();
        }
    }
    return e;
}

}  // namespace slsf
