/*
 * Sweeps and measurements of lattices held in global memory, L_x a multiple
 * of 4, walked along z in patches (walk.cuh): the single-task calls, the large
 * lattices of a batch and, many replicas per launch, the replicas too large
 * for one CTA's shared memory.
 *
 *   k_walk_colour   one colour of metropolis_sweep_with_scratch
 *                   (src/updates.rs:440-486); colour 0 optionally fused with
 *                   the measurement of the state it starts from
 *   k_walk_measure  measure_theta_observables_with_scratch
 *                   (src/observables.rs:80-154)
 *
 * A thread reads the four sites x = 4 q .. 4 q + 3 of a row with one 16-byte
 * load (the angles are one 256-byte aligned array and L_x is a multiple of 4)
 * and gets a pair of each colour.  A colour's kernel writes only that colour;
 * its 16-byte stores put back the other colour's words as they were, which no
 * thread of the launch changes.
 */
#include <algorithm>

#include "engine.h"
#include "walk.cuh"
#include "xy_device.cuh"

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

/* The block's sums to the replica's partials; the last of its `blocks` blocks
 * adds the partials in block order, writes the totals and adds the measured
 * values to bin_row (NULL: none) in the batched kernels' column order
 * (ThetaModel::measure's stream, src/model.rs:406-409). */
__device__ __forceinline__ void finish_sums(double (&acc)[8], const TaskView& t, uint32_t blocks, double* bin_row) {
    __shared__ double scratch[8 * 32];
    __shared__ bool last;
    block_sum<8>(acc, scratch);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) t.partials[blockIdx.x * 8 + k] = acc[k];
        __threadfence();
        last = atomicAdd(t.done, 1u) == blocks - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < blocks; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < 8; ++k) tot[k] += __ldcg(&t.partials[b * 8 + k]);
    block_sum<8>(tot, scratch);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) t.result[k] = tot[k];
        if (bin_row) {
            const double v = (double)(t.lx * t.ly * t.lz);
            const double e = -(tot[2] + tot[3] + tot[4]) / v;
            const double vals[kBinCols] = {e,      e * e,  (tot[0] * tot[0] + tot[1] * tot[1]) / (v * v),
                                           tot[2], tot[3], tot[4],
                                           tot[5], tot[6], tot[7],
                                           tot[5] * tot[5], tot[6] * tot[6], tot[7] * tot[7]};
            for (int q = 0; q < kBinCols; ++q) bin_row[q] += vals[q];
        }
        *t.done = 0;
    }
}

/* Bin row of the state after `done` sweeps, NULL if it is not measured or kept. */
__device__ __forceinline__ double* bin_row_of(const TaskView& t, uint64_t done) {
    if (t.n_bins == 0 || done <= t.thermalization) return nullptr;
    const uint64_t b = (done - t.thermalization - 1) / t.binsize;
    return b < t.n_bins ? t.bins + b * kBinCols : nullptr;
}

/* A thread's patch of rows y0, y0 + 1 (y0 even) by x = 4 q .. 4 q + 3 for the
 * planes z_lo .. z_hi - 1 of the replica. */
struct Patch {
    uint32_t y0, q, z_lo, z_hi;
};

__device__ __forceinline__ bool patch_of(const TaskView& t, uint32_t unit, uint32_t seglen, Patch& p) {
    const uint32_t nq = t.lx >> 2, ncol = nq * (t.ly >> 1);
    const uint32_t sg = unit / ncol, col = unit - sg * ncol, m = col / nq;
    p.q = col - m * nq;
    p.y0 = 2u * m;
    p.z_lo = sg * seglen;
    p.z_hi = min(t.lz, p.z_lo + seglen);
    return p.z_lo < t.lz;
}

__host__ __device__ inline uint32_t walk_blocks(const TaskView& t, uint32_t seglen) {
    const uint32_t ncol = (t.lx >> 2) * (t.ly >> 1), nseg = (t.lz + seglen - 1) / seglen;
    return (ncol * nseg + kWalkThreads - 1) / kWalkThreads;
}

/* One colour.  Bound by instruction issue (two Philox blocks, 14 neighbour
 * and 8 own sincos per four updates); angles come from L2 or HBM, 12 bytes
 * per update. */
template <bool kMeasure>
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocksPerSm)
    k_walk_colour(const TaskView* __restrict__ views, TaskView one, const unsigned long long* __restrict__ counters,
                  uint32_t sw, uint32_t colour, uint32_t seglen, double* one_bin_row) {
    const TaskView t = views ? views[blockIdx.y] : one;
    if (views && sw >= t.sweeps) return;
    const uint32_t blocks = walk_blocks(t, seglen);
    if (blockIdx.x >= blocks) return;
    const uint64_t sweep = (counters ? counters[2 * blockIdx.y] : t.metro_sweeps) + sw;
    const uint32_t lx = t.lx, plane = lx * t.ly;
    uint32_t accepted = 0;
    /* each of a thread's sums takes four terms per plane, at most 1 or J in magnitude */
    const float bias = 8.0f * (float)seglen;
    Sum2 sum[kMeasure ? 8 : 1];
    if (kMeasure)
#pragma unroll
        for (int k = 0; k < 8; ++k) sum[k].start(k < 2 ? bias : t.jmax * bias);
    Patch pt;
    if (patch_of(t, blockIdx.x * kWalkThreads + threadIdx.x, seglen, pt)) {
        float* th = t.theta;
        const float *jxy = t.jxy, *jz = t.jz;
        /* offsets in a plane: the patch's rows, the rows below and above, the x neighbours left and right */
        const uint32_t i0 = pt.y0 * lx + 4u * pt.q, i1 = i0 + lx;
        const uint32_t im = (pt.y0 == 0 ? t.ly - 1 : pt.y0 - 1) * lx + 4u * pt.q;
        const uint32_t ip = (pt.y0 + 2 == t.ly ? 0u : pt.y0 + 2) * lx + 4u * pt.q;
        const uint32_t xl = pt.q == 0 ? i0 + lx - 1 : i0 - 1, xr = 4u * pt.q + 4 == lx ? pt.y0 * lx : i0 + 4;
        auto four = [&](uint32_t at) { return *reinterpret_cast<const float4*>(th + at); };
        /* the sites x = 4 q + par, 4 q + 2 + par of four */
        auto pick = [](const float4& v, bool par) { return par ? make_float2(v.y, v.w) : make_float2(v.x, v.z); };
        auto trig1 = [&](uint32_t at) {
            float sn, cn;
            __sincosf(th[at], &sn, &cn);
            return make_float2(cn, sn);
        };
        uint32_t base = pt.z_lo * plane;
        const uint32_t below = (pt.z_lo == 0 ? t.lz - 1 : pt.z_lo - 1) * plane;
        /* the parity of row y0 in plane z: its own colour at x = 2 k + parity, the other at 2 k + 1 - parity */
        const bool par_lo = (colour + pt.z_lo) & 1u;
        float4 r0 = four(base + i0), r1 = four(base + i1); /* this plane's rows */
        Trig2 m0 = trig2(pick(four(below + i0), par_lo)), m1 = trig2(pick(four(below + i1), !par_lo));
        Trig2 c0 = trig2(pick(r0, !par_lo)), c1 = trig2(pick(r1, par_lo));
        float jzm = jz[pt.z_lo == 0 ? t.lz - 1 : pt.z_lo - 1];
        auto step = [&](uint32_t z, auto odd) {
            constexpr bool kOdd = decltype(odd)::value;
            const uint32_t above = z + 1 == t.lz ? 0u : base + plane;
            const float4 n0 = four(above + i0), n1 = four(above + i1);
            const float4 vm = four(base + im), vp = four(base + ip);
            const float2 e0 = trig1(base + (kOdd ? xr : xl)), e1 = trig1(base + lx + (kOdd ? xl : xr));
            const float jx = jxy[z], jzp = jz[z];
            const uint32_t unit = (base + i0) >> 2;
            const slsf_u32x4 b0 = slsf_stream(t.seed, sweep, SLSF_PURPOSE_METRO, colour, unit);
            const slsf_u32x4 b1 = slsf_stream(t.seed, sweep, SLSF_PURPOSE_METRO, colour, unit + (lx >> 2));
            const Trig2 p0 = trig2(pick(n0, kOdd)), p1 = trig2(pick(n1, !kOdd));
            const Trig2 ym = trig2(pick(vm, kOdd)), yp = trig2(pick(vp, !kOdd));
            float2 own = pick(r0, kOdd);
            accepted += update_pair<kMeasure, kOdd>(own, c0, e0, ym, c1, m0, p0, jx, jzp, jzm, t.beta, t.width, b0, sum);
            (kOdd ? r0.y : r0.x) = own.x;
            (kOdd ? r0.w : r0.z) = own.y;
            *reinterpret_cast<float4*>(th + base + i0) = r0;
            own = pick(r1, !kOdd);
            accepted += update_pair<kMeasure, !kOdd>(own, c1, e1, c0, yp, m1, p1, jx, jzp, jzm, t.beta, t.width, b1, sum);
            (kOdd ? r1.x : r1.y) = own.x;
            (kOdd ? r1.z : r1.w) = own.y;
            *reinterpret_cast<float4*>(th + base + i1) = r1;
            m0 = c0;
            m1 = c1;
            c0 = p0;
            c1 = p1;
            r0 = n0;
            r1 = n1;
            jzm = jzp;
            base += plane;
        };
        uint32_t z = pt.z_lo;
        if (par_lo) step(z++, std::true_type());
        for (; z + 1 < pt.z_hi; z += 2) {
            step(z, std::false_type());
            step(z + 1, std::true_type());
        }
        if (z < pt.z_hi) step(z, std::false_type());
    }
    block_count(accepted, t.stats, kStatAccepted);
    if (kMeasure) {
        double acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = sum[k].total(k < 2 ? bias : t.jmax * bias);
        double* row = views ? (sw > 0 ? bin_row_of(t, sweep) : nullptr) : one_bin_row;
        finish_sums(acc, t, blocks, row);
    }
}

/* J cos and J sin of the bonds a -> b of two sites. */
__device__ __forceinline__ void add_bond2(Sum2& ac, Sum2& as, float j, const Trig2& a, const Trig2& b) {
    ac.add(__fmul2_rn(dup2(j), __ffma2_rn(a.c, b.c, __fmul2_rn(a.s, b.s))));
    as.add(__fmul2_rn(dup2(j), __ffma2_rn(a.s, b.c, __fmul2_rn(neg2(a.c), b.s))));
}

/* The observables of the state, after its last sweep in a batched launch: 14
 * sincos per eight sites.  The sums in FP32 value and remainder (Sum2) instead
 * of FP64 conversions on the special-function pipe, which bound the earlier
 * row walk (72% of it busy, 86 us at L = 256). */
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocksPerSm)
    k_walk_measure(const TaskView* __restrict__ views, TaskView one, const unsigned long long* __restrict__ counters,
                   uint32_t seglen, double* one_bin_row) {
    const TaskView t = views ? views[blockIdx.y] : one;
    const uint32_t blocks = walk_blocks(t, seglen);
    if (blockIdx.x >= blocks) return;
    double* row = one_bin_row;
    if (views) {
        row = bin_row_of(t, (counters ? counters[2 * blockIdx.y] : t.metro_sweeps) + t.sweeps);
        if (!row) return;
    }
    const uint32_t lx = t.lx, plane = lx * t.ly;
    const float bias = 8.0f * (float)seglen;
    Sum2 sum[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[k].start(k < 2 ? bias : t.jmax * bias);
    Patch pt;
    if (patch_of(t, blockIdx.x * kWalkThreads + threadIdx.x, seglen, pt)) {
        const float* th = t.theta;
        const uint32_t i0 = pt.y0 * lx + 4u * pt.q, i1 = i0 + lx;
        const uint32_t ip = (pt.y0 + 2 == t.ly ? 0u : pt.y0 + 2) * lx + 4u * pt.q;
        const uint32_t xr = 4u * pt.q + 4 == lx ? pt.y0 * lx : i0 + 4;
        struct Quad {
            Trig2 a, b; /* sites 0, 1 and 2, 3 */
        };
        auto quad = [&](uint32_t at) {
            const float4 v = *reinterpret_cast<const float4*>(th + at);
            Quad r;
            r.a = trig2(make_float2(v.x, v.y));
            r.b = trig2(make_float2(v.z, v.w));
            return r;
        };
        auto xnext = [&](const Quad& c, uint32_t at) { /* the four +x neighbours */
            float sn, cn;
            __sincosf(th[at], &sn, &cn);
            Quad r;
            r.a.c = make_float2(c.a.c.y, c.b.c.x);
            r.a.s = make_float2(c.a.s.y, c.b.s.x);
            r.b.c = make_float2(c.b.c.y, cn);
            r.b.s = make_float2(c.b.s.y, sn);
            return r;
        };
        uint32_t base = pt.z_lo * plane;
        Quad c0 = quad(base + i0), c1 = quad(base + i1);
        for (uint32_t z = pt.z_lo; z < pt.z_hi; ++z) {
            const uint32_t above = z + 1 == t.lz ? 0u : base + plane;
            const Quad n0 = quad(above + i0), n1 = quad(above + i1), yp = quad(base + ip);
            const Quad x0 = xnext(c0, base + xr), x1 = xnext(c1, base + lx + xr);
            const float jx = t.jxy[z], jzz = t.jz[z];
            auto site = [&](const Trig2& i, const Trig2& xp, const Trig2& up, const Trig2& zp) {
                sum[0].add(i.c);
                sum[1].add(i.s);
                add_bond2(sum[2], sum[5], jx, i, xp);
                add_bond2(sum[3], sum[6], jx, i, up);
                add_bond2(sum[4], sum[7], jzz, i, zp);
            };
            site(c0.a, x0.a, c1.a, n0.a);
            site(c0.b, x0.b, c1.b, n0.b);
            site(c1.a, x1.a, yp.a, n1.a);
            site(c1.b, x1.b, yp.b, n1.b);
            c0 = n0;
            c1 = n1;
            base += plane;
        }
    }
    double acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = sum[k].total(k < 2 ? bias : t.jmax * bias);
    finish_sums(acc, t, blocks, row);
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

bool walk_supports(const TaskView& t) {
    /* patches of four sites by two rows; the biased sums need finite couplings; 32-bit site indices; a block sum per
     * block of the partials' rows */
    return t.lx % 4 == 0 && t.ly % 2 == 0 && t.lz >= 2 && t.jmax < kJMax &&
           (reinterpret_cast<uintptr_t>(t.theta) & 15u) == 0 && (uint64_t)t.lx * t.ly * t.lz <= 0x7fffffffull &&
           walk_blocks(t, t.lz) <= (uint32_t)kMeasureMaxBlocks;
}

uint32_t walk_seglen(const TaskView& t, uint32_t n) {
    /* Planes per thread: as many segments as fill one, two, three or four
     * rounds of the resident blocks, whichever ends first when a round takes its
     * planes and about 0.7 of a plane to fill the window; at least two planes.
     * (L = 256: 29 planes, 288 blocks on 296 places; L = 64: two, 64 blocks.) */
    const uint64_t places = (uint64_t)sm_count() * kWalkBlocksPerSm, ncol = (uint64_t)(t.lx >> 2) * (t.ly >> 1);
    uint32_t best = t.lz;
    double cost = 1e300;
    for (uint32_t r = 1; r <= 4; ++r) {
        const uint64_t blocks = std::min<uint64_t>(std::max<uint64_t>(r * places / n, 1), kMeasureMaxBlocks);
        const uint64_t nseg = std::min<uint64_t>(std::max<uint64_t>(blocks * kWalkThreads / ncol, 1), std::max(1u, t.lz / 2));
        const uint32_t len = (uint32_t)((t.lz + nseg - 1) / nseg);
        const double rounds = (double)((walk_blocks(t, len) * (uint64_t)n + places - 1) / places);
        if (rounds * (len + 0.7) < cost) {
            cost = rounds * (len + 0.7);
            best = len;
        }
    }
    return best;
}

void launch_walk_colour(const TaskView& t, uint64_t sweep, uint32_t colour, bool measure, double* bin_row, cudaStream_t s) {
    TaskView v = t;
    v.metro_sweeps = sweep;
    const uint32_t len = walk_seglen(v, 1);
    if (measure)
        k_walk_colour<true><<<walk_blocks(v, len), kWalkThreads, 0, s>>>(nullptr, v, nullptr, 0, colour, len, bin_row);
    else
        k_walk_colour<false><<<walk_blocks(v, len), kWalkThreads, 0, s>>>(nullptr, v, nullptr, 0, colour, len, nullptr);
}

void launch_walk_measure(const TaskView& t, double* bin_row, cudaStream_t s) {
    const uint32_t len = walk_seglen(t, 1);
    k_walk_measure<<<walk_blocks(t, len), kWalkThreads, 0, s>>>(nullptr, t, nullptr, len, bin_row);
}

}  // namespace slsf
