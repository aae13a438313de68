/*
 * Batched persistent kernel for replicas that fit in one CTA's shared
 * memory: many replicas of uneven size, one CTA per replica at a time, each
 * replica resident for all of its sweeps.  Replaces the carlo-mc Runner's
 * task-by-task loop over ThetaModel::sweep + ThetaModel::measure
 * (src/model.rs:379-442, src/results.rs:200-202) for every task of a batch.
 *
 * Per replica the CTA
 *   1. copies theta from HBM into a colour-split shared layout: the colour-c
 *      site with index idx sits at c * (V/2 + 16) + idx/2, so a warp reading
 *      one colour reads consecutive words, and the 64-byte pad puts the two
 *      colours of neighbouring sites in different bank halves;
 *   2. per sweep: two colour half-sweeps (the same decision code as the
 *      single-task kernel, xy_device.cuh) and `wolff_steps` Wolff updates;
 *      after thermalization each sweep's state is measured inside the next
 *      sweep's colour-0 half-sweep (the launch's last state by a separate
 *      pass) and added to the task's bins;
 *   3. copies theta back.
 * HBM traffic is 8 bytes per site per launch, independent of the sweep
 * count.  Trig values are recomputed with __sincosf where needed (a 32^3
 * replica leaves no room for a cos/sin cache next to theta).
 *
 * Wolff labelling is bit-parallel: the active +x/+y/+z bonds of a row of
 * L_x <= 32 sites are three 32-bit words; the cluster grows from the seed by
 * OR-ing neighbour rows through the bond words and closing every row that
 * gained bits along x, until a pass changes nothing: three steps of every row
 * and one block barrier a pass, which for replicas of this size beats scans of
 * whole lines (grow, below).  The result is the seed's
 * connected component over the active bonds -- the set the reference's DFS
 * (src/updates.rs:577-597) collects when fed the same per-bond randoms.
 * Growth is monotone, so the pass count is bounded by V.
 */
#include <algorithm>
#include <type_traits>

#include "bins.cuh"
#include "bitgrow.cuh"
#include "engine.h"
#include "fastdiv.h"
#include "walk.cuh"
#include "xy_device.cuh"

namespace slsf {

namespace {

constexpr int kBThreads = 1024;
constexpr uint32_t kPad = 16; /* floats: 64 bytes */
constexpr uint32_t kMaxRowBits = 32;

/* Optional per-phase cycle accounting (build with -DSLSF_PHASE_TIMING):
 * thread 0 of every CTA adds the clock64 cycles of each phase, measured
 * between block barriers, to g_phase_cycles; slot 6 counts cluster-growth
 * passes and slot 7 Wolff updates. */
#ifdef SLSF_PHASE_TIMING
__device__ unsigned long long g_res_phase_cycles[8];
__shared__ long long s_phase_mark;
#define SLSF_PHASE(k)                                                                     \
    do {                                                                                  \
        __syncthreads();                                                                  \
        if (threadIdx.x == 0) {                                                           \
            const long long now_ = clock64();                                             \
            atomicAdd(&g_res_phase_cycles[k], (unsigned long long)(now_ - s_phase_mark)); \
            s_phase_mark = now_;                                                          \
        }                                                                                 \
    } while (0)
#define SLSF_PHASE_COUNT(k, n)                                                              \
    do {                                                                                    \
        if (threadIdx.x == 0) atomicAdd(&g_res_phase_cycles[k], (unsigned long long)(n)); \
    } while (0)
#else
#define SLSF_PHASE(k) \
    do {              \
    } while (0)
#define SLSF_PHASE_COUNT(k, n) \
    do {                       \
    } while (0)
#endif

struct Geo {
    uint32_t lx, ly, lz, volume, half, rows, plane;
    uint32_t stride1; /* offset of the colour-1 array */
    uint32_t xmask;
    bool lx_tiles_warp;
    slsf_fastdiv div_hx, div_ly, div_lx, div_nq;
};

__device__ __forceinline__ Geo make_geo(const TaskView& t) {
    Geo g;
    g.lx = t.lx;
    g.ly = t.ly;
    g.lz = t.lz;
    g.plane = t.lx * t.ly;
    g.volume = g.plane * t.lz;
    g.half = g.volume >> 1;
    g.rows = t.ly * t.lz;
    g.stride1 = g.half + kPad;
    g.xmask = t.lx >= 32 ? 0xffffffffu : ((1u << t.lx) - 1u);
    g.lx_tiles_warp = (32u % t.lx) == 0;
    g.div_hx = slsf_fastdiv_make(t.lx >> 1);
    g.div_ly = slsf_fastdiv_make(t.ly);
    g.div_lx = slsf_fastdiv_make(t.lx);
    g.div_nq = slsf_fastdiv_make(max(1u, t.lx >> 2));
    return g;
}

/* Shared-memory slot of natural site index idx with colour c. */
__device__ __forceinline__ uint32_t slot(const Geo& g, uint32_t idx, uint32_t colour) {
    return colour * g.stride1 + (idx >> 1);
}

struct Coords {
    uint32_t x, y, z, row;
};

__device__ __forceinline__ Coords coords_of(const Geo& g, uint32_t idx) {
    Coords c;
    c.row = slsf_fastdiv_div(idx, g.div_lx);
    c.x = idx - c.row * g.lx;
    c.z = slsf_fastdiv_div(c.row, g.div_ly);
    c.y = c.row - c.z * g.ly;
    return c;
}

/* Forward neighbours of a site (+x, +y, +z) as natural indices. */
__device__ __forceinline__ void forward_neighbours(const Geo& g, uint32_t idx, const Coords& c, uint32_t& xp,
                                                   uint32_t& yp, uint32_t& zp) {
    xp = (c.x + 1 == g.lx) ? idx + 1 - g.lx : idx + 1;
    yp = (c.y + 1 == g.ly) ? idx + g.lx - g.plane : idx + g.lx;
    zp = (c.z + 1 == g.lz) ? idx + g.plane - g.volume : idx + g.plane;
}

/* Row word of row y of plane z (the bond and cluster words). */
__device__ __forceinline__ uint32_t row_word(const Geo& g, uint32_t y, uint32_t z) { return y + g.ly * z; }

/* Lane holding the +x neighbour when rows of lx sites tile the warp. */
__device__ __forceinline__ uint32_t xp_lane(uint32_t lane, uint32_t lx) {
    return (lane & ~(lx - 1u)) | ((lane + 1u) & (lx - 1u));
}

struct Smem {
    float* th; /* two colour arrays */
    uint32_t* bx;
    uint32_t* by;
    uint32_t* bz;
    uint32_t* cl;
    float* jxy;
    float* jz;
    double* corr;  /* fused correlation scratch (resident_corr_doubles) */
};

__device__ __forceinline__ Smem carve(unsigned char* base, uint32_t max_volume, uint32_t max_rows, uint32_t max_lz) {
    Smem s;
    s.th = reinterpret_cast<float*>(base);
    uint32_t* w = reinterpret_cast<uint32_t*>(base + 4ull * (max_volume + 2 * kPad));
    s.bx = w;
    s.by = w + max_rows;
    s.bz = w + 2 * max_rows;
    s.cl = w + 3 * max_rows;
    s.jxy = reinterpret_cast<float*>(w + 4 * max_rows);
    s.jz = s.jxy + max_lz;
    /* 8-byte aligned: the volume is even, the other arrays are whole words */
    s.corr = reinterpret_cast<double*>(s.jz + max_lz);
    return s;
}

/* ---- phases ---- */

__device__ __forceinline__ void load_state(const TaskView& t, const Geo& g, Smem& s) {
    if (g.lx % 4) {
        /* L_x = 2 mod 4: four consecutive sites may span two rows; copy site by site */
        for (uint32_t i = threadIdx.x; i < g.volume; i += blockDim.x) {
            const Coords c = coords_of(g, i);
            s.th[slot(g, i, (c.x + c.y + c.z) & 1u)] = t.theta[i];
        }
    } else {
        const float4* src = reinterpret_cast<const float4*>(t.theta);
        for (uint32_t q = threadIdx.x; q < g.volume / 4; q += blockDim.x) {
            const float4 v = src[q];
            const Coords c = coords_of(g, 4 * q);
            const uint32_t p = (c.y + c.z) & 1u; /* colour of the even-x site */
            const uint32_t h = 2 * q;
            s.th[p * g.stride1 + h] = v.x;
            s.th[(p ^ 1u) * g.stride1 + h] = v.y;
            s.th[p * g.stride1 + h + 1] = v.z;
            s.th[(p ^ 1u) * g.stride1 + h + 1] = v.w;
        }
    }
    for (uint32_t z = threadIdx.x; z < g.lz; z += blockDim.x) {
        s.jxy[z] = t.jxy[z];
        s.jz[z] = t.jz[z];
    }
}

__device__ __forceinline__ void store_state(const TaskView& t, const Geo& g, const Smem& s) {
    if (g.lx % 4) {
        for (uint32_t i = threadIdx.x; i < g.volume; i += blockDim.x) {
            const Coords c = coords_of(g, i);
            t.theta[i] = s.th[slot(g, i, (c.x + c.y + c.z) & 1u)];
        }
        return;
    }
    float4* dst = reinterpret_cast<float4*>(t.theta);
    for (uint32_t q = threadIdx.x; q < g.volume / 4; q += blockDim.x) {
        const Coords c = coords_of(g, 4 * q);
        const uint32_t p = (c.y + c.z) & 1u;
        const uint32_t h = 2 * q;
        dst[q] = make_float4(s.th[p * g.stride1 + h], s.th[(p ^ 1u) * g.stride1 + h], s.th[p * g.stride1 + h + 1],
                             s.th[(p ^ 1u) * g.stride1 + h + 1]);
    }
}

/* One colour half-sweep.  A warp owns 32 consecutive Philox blocks (64
 * sites); lanes exchange words so that lane j updates colour-compact sites
 * 2*base + j and 2*base + 32 + j, i.e. consecutive shared words.
 *
 * With kMeasure (colour 0 only) it also measures the state the half-sweep
 * starts from, at no extra trig: every bond joins a colour-0 site to a
 * colour-1 site, and before its update a colour-0 site has the trig of
 * itself and of all six neighbours, so it adds the terms of its three
 * forward bonds and of the three backward bonds that end on it, and the
 * magnetisation of itself and of its +x neighbour (each colour-1 site is the
 * +x neighbour of exactly one colour-0 site).  Each term is the bond_cos /
 * bond_sin value the measurement pass computes; sums are FP64. */
template <bool kMeasure>
__device__ __forceinline__ uint32_t half_sweep(const TaskView& t, const Geo& g, Smem& s, uint64_t sweep,
                                               uint32_t colour, double (&acc)[8]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t nwarps = blockDim.x >> 5;
    const uint32_t npairs = (g.half + 1) >> 1;
    const uint32_t own = colour * g.stride1, other = (colour ^ 1u) * g.stride1;
    uint32_t accepted = 0;
    for (uint32_t base = warp * 32; base < npairs; base += nwarps * 32) {
        const uint32_t p = base + lane;
        slsf_u32x4 blk = {0, 0, 0, 0};
        if (p < npairs) blk = slsf_stream(t.seed, sweep, SLSF_PURPOSE_METRO, colour, p);
#pragma unroll
        for (uint32_t r = 0; r < 2; ++r) {
            const uint32_t src = 16 * r + (lane >> 1);
            const uint32_t wx = __shfl_sync(0xffffffffu, blk.x, src);
            const uint32_t wy = __shfl_sync(0xffffffffu, blk.y, src);
            const uint32_t wz = __shfl_sync(0xffffffffu, blk.z, src);
            const uint32_t ww = __shfl_sync(0xffffffffu, blk.w, src);
            const uint32_t h = 2 * base + 32 * r + lane;
            if (h >= g.half) continue;
            const float u_prop = slsf_u24f((lane & 1u) ? wz : wx);
            const float u_acc = slsf_u24f((lane & 1u) ? ww : wy);
            const uint32_t row = slsf_fastdiv_div(h, g.div_hx);
            const uint32_t k = h - row * (g.lx >> 1);
            const uint32_t z = slsf_fastdiv_div(row, g.div_ly);
            const uint32_t y = row - z * g.ly;
            SiteXYZ st;
            st.x = 2u * k + ((colour + y + z) & 1u);
            st.y = y;
            st.z = z;
            st.idx = st.x + g.lx * row;
            uint32_t nb[6];
            neighbour_indices(st, g.lx, g.ly, g.lz, nb);
            const float jx = s.jxy[z], jzp = s.jz[z], jzm = s.jz[z == 0 ? g.lz - 1 : z - 1];
            const float th = s.th[own + h];
            float si, ci;
            __sincosf(th, &si, &ci);
            /* neighbours in pairs, folded into the field as they come */
            float sa, ca, sb, cb;
            __sincosf(s.th[other + (nb[0] >> 1)], &sa, &ca);
            __sincosf(s.th[other + (nb[1] >> 1)], &sb, &cb);
            if (kMeasure) {
                /* forward bonds i -> i+mu, backward bonds i-mu -> i */
                acc[0] += (double)ci + (double)ca;
                acc[1] += (double)si + (double)sa;
                acc[2] += (double)bond_cos(jx, ci, si, ca, sa) + (double)bond_cos(jx, cb, sb, ci, si);
                acc[5] += (double)bond_sin(jx, ci, si, ca, sa) + (double)bond_sin(jx, cb, sb, ci, si);
            }
            const float hx01 = __fadd_rn(ca, cb), hy01 = __fadd_rn(sa, sb);
            __sincosf(s.th[other + (nb[2] >> 1)], &sa, &ca);
            __sincosf(s.th[other + (nb[3] >> 1)], &sb, &cb);
            if (kMeasure) {
                acc[3] += (double)bond_cos(jx, ci, si, ca, sa) + (double)bond_cos(jx, cb, sb, ci, si);
                acc[6] += (double)bond_sin(jx, ci, si, ca, sa) + (double)bond_sin(jx, cb, sb, ci, si);
            }
            const float hx23 = __fadd_rn(ca, cb), hy23 = __fadd_rn(sa, sb);
            __sincosf(s.th[other + (nb[4] >> 1)], &sa, &ca);
            __sincosf(s.th[other + (nb[5] >> 1)], &sb, &cb);
            if (kMeasure) {
                acc[4] += (double)bond_cos(jzp, ci, si, ca, sa) + (double)bond_cos(jzm, cb, sb, ci, si);
                acc[7] += (double)bond_sin(jzp, ci, si, ca, sa) + (double)bond_sin(jzm, cb, sb, ci, si);
            }
            const float hx = field_from_pairs(jx, jzp, jzm, hx01, hx23, ca, cb);
            const float hy = field_from_pairs(jx, jzp, jzm, hy01, hy23, sa, sb);
            float tn, sn, cn;
            if (metro_decide(th, ci, si, hx, hy, t.beta, t.width, u_prop, u_acc, &tn, &sn, &cn)) {
                s.th[own + h] = tn;
                ++accepted;
            }
        }
    }
    return accepted;
}

/* The same colour half-sweep for L_x a multiple of 4, walking along z.  A
 * thread owns a patch of two rows (y0, y0 + 1; y0 even) by two compact sites
 * of each colour (k = 2 q, 2 q + 1, i.e. x = 4 q .. 4 q + 3) for a run of
 * planes and updates its four colour-c sites of a plane together:
 *   - it keeps the trig of the other colour's patch on the planes below, at
 *     and above (the z neighbours), which is also one x neighbour, the inner
 *     x neighbour of each pair and the inner y neighbours, so a plane takes 14
 *     neighbour sincos for four updates instead of 24, and no shuffles;
 *   - the two sites of a pair (h even, h + 1) share a Philox block, so a
 *     thread uses its two blocks per plane whole, with one key schedule;
 *   - the pair's arithmetic is packed (two FP32 operations per instruction);
 *   - y0 is even, so the rows' parities depend on the plane alone and the
 *     planes are unrolled by two instead of selecting by parity.
 * The kernel is bound by instruction issue; the earlier form (one site per
 * lane, x neighbours by shuffle, L_x = 32 only) took 186 instructions per
 * update.  Operands, rounding order and randoms are those of half_sweep, so
 * decisions and new angles are bit-identical. */
template <bool kMeasure>
__device__ __forceinline__ uint32_t half_sweep_quads(const TaskView& t, const Geo& g, Smem& s, uint64_t sweep,
                                                     uint32_t colour, double (&acc)[8]) {
    const uint32_t hx = g.lx >> 1, nq = g.lx >> 2, ncol = nq * (g.ly >> 1), plane = hx * g.ly;
    /* planes per unit: every thread gets work when there are fewer patches than threads */
    const uint32_t nseg = max(1u, min(g.lz >> 1, blockDim.x / ncol));
    const uint32_t seglen = (g.lz + nseg - 1) / nseg;
    float* own = s.th + colour * g.stride1;
    const float* oth = s.th + (colour ^ 1u) * g.stride1;
    uint32_t accepted = 0;
    WalkSums sums;
    if (kMeasure) sums.start(t.jxy_max, t.jz_max);
    Sum2* sum = kMeasure ? sums.run : nullptr;
    for (uint32_t u = threadIdx.x; u < ncol * nseg; u += blockDim.x) {
        const uint32_t sg = u / ncol, col = u - sg * ncol, m = col / nq, q = col - m * nq;
        const uint32_t z_lo = sg * seglen, z_hi = min(g.lz, z_lo + seglen);
        if (z_lo >= z_hi) continue;
        const uint32_t y0 = 2u * m;
        /* compact offsets in a plane: the patch's rows, the rows below and above, the x neighbours left and right */
        const uint32_t h0 = y0 * hx + 2u * q, h1 = h0 + hx;
        const uint32_t hm = (y0 == 0 ? g.ly - 1 : y0 - 1) * hx + 2u * q;
        const uint32_t hp = (y0 + 2 == g.ly ? 0u : y0 + 2) * hx + 2u * q;
        const uint32_t xl = q == 0 ? h0 + hx - 1 : h0 - 1, xr = q + 1 == nq ? h0 + 2 - hx : h0 + 2;
        auto two = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
        auto trig1 = [&](uint32_t at) {
            float sn, cn;
            __sincosf(oth[at], &sn, &cn);
            return make_float2(cn, sn);
        };
        uint32_t base = z_lo * plane;
        const uint32_t below = (z_lo == 0 ? g.lz - 1 : z_lo - 1) * plane;
        Trig2 m0 = trig2(two(oth + below + h0)), m1 = trig2(two(oth + below + h1)); /* plane below */
        Trig2 c0 = trig2(two(oth + base + h0)), c1 = trig2(two(oth + base + h1));   /* this plane */
        float jzm = s.jz[z_lo == 0 ? g.lz - 1 : z_lo - 1];
        /* one plane; kOdd: the parity (colour + y0 + z) & 1 of row y0, whose colour-c sites sit at x = 2 k + parity */
        auto step = [&](uint32_t z, auto odd) {
            constexpr bool kOdd = decltype(odd)::value;
            const uint32_t above = z + 1 == g.lz ? 0u : base + plane;
            const Trig2 p0 = trig2(two(oth + above + h0)), p1 = trig2(two(oth + above + h1));
            const float jx = s.jxy[z], jzp = s.jz[z];
            const Trig2 ym = trig2(two(oth + base + hm)), yp = trig2(two(oth + base + hp));
            const float2 e0 = trig1(base + (kOdd ? xr : xl)), e1 = trig1(base + hx + (kOdd ? xl : xr));
            const uint32_t unit = (base + h0) >> 1;
            const slsf_u32x4 b0 = slsf_stream(t.seed, sweep, SLSF_PURPOSE_METRO, colour, unit);
            const slsf_u32x4 b1 = slsf_stream(t.seed, sweep, SLSF_PURPOSE_METRO, colour, unit + (hx >> 1));
            auto row = [&](uint32_t h, const Trig2& c, float2 e, auto row_odd, const Trig2& dn, const Trig2& up,
                           const Trig2& zm, const Trig2& zp, const slsf_u32x4& b) {
                float2 th = two(own + base + h);
                accepted += update_pair<kMeasure, decltype(row_odd)::value>(th, c, e, dn, up, zm, zp, jx, jzp, jzm,
                                                                            t.beta, t.width, b, sum);
                *reinterpret_cast<float2*>(own + base + h) = th;
            };
            row(h0, c0, e0, std::integral_constant<bool, kOdd>(), ym, c1, m0, p0, b0);
            row(h1, c1, e1, std::integral_constant<bool, !kOdd>(), c0, yp, m1, p1, b1);
            m0 = c0;
            m1 = c1;
            c0 = p0;
            c1 = p1;
            jzm = jzp;
            base += plane;
        };
        uint32_t z = z_lo;
        bool open = false; /* terms that are not in the FP64 sums yet */
        if ((colour + z) & 1u) {
            step(z++, std::true_type());
            open = true;
        }
        for (; z + 1 < z_hi; z += 2) {
            step(z, std::false_type());
            step(z + 1, std::true_type());
            if (kMeasure) sums.flush();
            open = false;
        }
        if (z < z_hi) {
            step(z, std::false_type());
            open = true;
        }
        if (kMeasure && open) sums.flush();
    }
    if (kMeasure)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += sums.acc[k];
    return accepted;
}

/* One colour half-sweep: the patch walk for L_x a multiple of 4, the
 * site-by-site form for L_x = 2 mod 4, whose pairs of compact sites straddle rows
 * (and for couplings whose biased sums could overflow).  The walk from 1,024
 * sites on, where its units fill the block: a thread
 * has at least one plane's four updates to do one after the other, and in a
 * smaller lattice that chain is longer than half_sweep's, with a site per lane
 * (us per sweep of 8 replicas alone, and of 2048 per 148 of them, walk and
 * half_sweep: 4^3 8.2 / 3.2 and 5.6 / 2.4, 8^3 9.3 / 3.8 and 8.5 / 3.2; 12^3
 * 13.3 / 7.4 and 27.7 / 9.5). */
constexpr uint32_t kQuadSites = 1024;

template <bool kMeasure>
__device__ __forceinline__ uint32_t sweep_colour(const TaskView& t, const Geo& g, Smem& s, uint64_t sweep,
                                                 uint32_t colour, double (&acc)[8]) {
    if (g.lx % 4 == 0 && g.volume >= kQuadSites && (!kMeasure || fmaxf(t.jxy_max, t.jz_max) < kJMax))
        return half_sweep_quads<kMeasure>(t, g, s, sweep, colour, acc);
    return half_sweep<kMeasure>(t, g, s, sweep, colour, acc);
}

__device__ __forceinline__ float site_theta(const Geo& g, const Smem& s, uint32_t idx, const Coords& c) {
    return s.th[slot(g, idx, (c.x + c.y + c.z) & 1u)];
}

/* Growth passes over row words: every row takes the cluster bits that reach
 * it through its y and z bonds; a row that gained bits is closed along x
 * (stored rows are always closed).  Rows updated earlier in the same pass are
 * seen by later ones, so bits can travel more than one row per pass. */
constexpr int kGrowSteps = 3; /* steps of every row between two block barriers */

/* One step of a row from the words around it; returns whether it changed. */
__device__ __forceinline__ bool grow_row(volatile uint32_t* cl, uint32_t w, uint32_t in, uint32_t bx, uint32_t lx) {
    const uint32_t old = cl[w], c = old | in;
    if (c == old) return false;
    cl[w] = close_word(c, bx, lx, true);
    return true;
}

/* R rows per thread, everything but the cluster words looked up once and
 * kept in registers.  A pass takes kGrowSteps steps of every row and one block
 * barrier with the vote: bits only ever get set, so a pass in which no row
 * changed saw the same words throughout and the cluster is closed. */
template <int R>
__device__ __forceinline__ uint32_t grow_rows(const Geo& g, Smem& s, uint32_t bound) {
    uint32_t w[R], yp[R], ym[R], zp[R], zm[R], b_yp[R], b_ym[R], b_zp[R], b_zm[R], b_x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const uint32_t r = threadIdx.x + k * blockDim.x;
        const bool has = r < g.rows;
        const uint32_t z = has ? slsf_fastdiv_div(r, g.div_ly) : 0u, y = has ? r - z * g.ly : 0u;
        w[k] = row_word(g, y, z);
        yp[k] = row_word(g, y + 1 == g.ly ? 0 : y + 1, z);
        ym[k] = row_word(g, y == 0 ? g.ly - 1 : y - 1, z);
        zp[k] = row_word(g, y, z + 1 == g.lz ? 0 : z + 1);
        zm[k] = row_word(g, y, z == 0 ? g.lz - 1 : z - 1);
        b_yp[k] = has ? s.by[w[k]] : 0u;
        b_ym[k] = has ? s.by[ym[k]] : 0u;
        b_zp[k] = has ? s.bz[w[k]] : 0u;
        b_zm[k] = has ? s.bz[zm[k]] : 0u;
        b_x[k] = s.bx[w[k]];
    }
    volatile uint32_t* cl = s.cl;
    for (uint32_t pass = 0; pass < bound; ++pass) {
        int changed = 0;
#pragma unroll 1
        for (int step = 0; step < kGrowSteps; ++step) {
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const uint32_t in = (cl[ym[k]] & b_ym[k]) | (cl[yp[k]] & b_yp[k]) | (cl[zm[k]] & b_zm[k]) |
                                    (cl[zp[k]] & b_zp[k]);
                if (grow_row(cl, w[k], in, b_x[k], g.lx)) changed = 1;
            }
        }
        if (!__syncthreads_or(changed)) return pass + 1;
    }
    return 0;
}

/* Grows the cluster (the closed seed row in cl) over the bond words; returns
 * the passes taken, 0 if they exceeded `bound`.  A barrier every three steps
 * against one every step takes a seventh off at L = 32 (18.4k -> 15.8k cycles
 * per update, 2: 16.2k, 4: 15.7k); up to four rows per thread stay in
 * registers (measured before, with words and divisions looked up in every
 * step: L = 16 24.0k -> 12.0k, L = 24 43.5k -> 25.0k).  Scans of whole lines by
 * shuffles need fewer passes (10 at L = 32) but longer ones: 17-19k cycles at
 * L = 32, 39k at L = 24, 35k at L = 16. */
__device__ __forceinline__ uint32_t grow(const Geo& g, Smem& s, uint32_t bound) {
    if (g.rows <= blockDim.x) return grow_rows<1>(g, s, bound);
    if (g.rows <= 2 * blockDim.x) return grow_rows<2>(g, s, bound);
    if (g.rows <= 4 * blockDim.x) return grow_rows<4>(g, s, bound);
    volatile uint32_t* cl = s.cl;
    for (uint32_t pass = 0; pass < bound; ++pass) {
        int changed = 0;
        for (uint32_t r = threadIdx.x; r < g.rows; r += blockDim.x) {
            const uint32_t z = slsf_fastdiv_div(r, g.div_ly), y = r - z * g.ly;
            const uint32_t ym = row_word(g, y == 0 ? g.ly - 1 : y - 1, z), zm = row_word(g, y, z == 0 ? g.lz - 1 : z - 1);
            const uint32_t in = (cl[ym] & s.by[ym]) | (cl[row_word(g, y + 1 == g.ly ? 0 : y + 1, z)] & s.by[r]) |
                                (cl[zm] & s.bz[zm]) | (cl[row_word(g, y, z + 1 == g.lz ? 0 : z + 1)] & s.bz[r]);
            if (grow_row(cl, r, in, s.bx[r], g.lx)) changed = 1;
        }
        if (!__syncthreads_or(changed)) return pass + 1;
    }
    return 0;
}

/* Bond activation: the +x, +y, +z bond words of every row.  A warp holds
 * G = 32 / L_x rows side by side (lane = x + L_x sub; the lanes past them keep
 * no bits), sub-group sub in the planes z = 2 (G zb + sub) and z + 1, and
 * walks columns of rows along y -- (zb, y segment) units, round robin.  The
 * +y row's projections are the next row's own and plane z's +z partner is
 * plane z + 1's site, so a step takes three sincos for its two sites; the two
 * sites' arithmetic is packed (two FP32 operations per instruction) and their
 * two Philox blocks share one key schedule.  Sub-groups past the last plane
 * compute on the last planes and keep nothing.  Bound by instruction issue:
 * one Philox block and three bond tests per site. */
template <int kUnroll>
__device__ __forceinline__ void wolff_bonds(const TaskView& t, const Geo& g, const Smem& s, uint64_t counter,
                                            float cphi, float sphi) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t groups = 32u / g.lx, sub = min(lane / g.lx, groups - 1), x = lane - sub * g.lx;
    const bool keep = x < g.lx;
    const uint32_t xl = keep ? x : 0u, hx = g.lx >> 1, ph = g.plane >> 1;
    const uint32_t nzb = ((g.lz >> 1) + groups - 1) / groups;
    /* runs of at most 32 rows: lane j keeps the ballots of the run's row j until its end */
    const uint32_t nseg = max(min(g.ly, (nwarps + nzb - 1) / nzb), (g.ly + 31u) >> 5);
    const uint32_t seg = (g.ly + nseg - 1) / nseg;
    const uint32_t xsrc = sub * g.lx + (xl + 1 == g.lx ? 0u : xl + 1);
    const float2 cphi2 = make_float2(cphi, cphi), sphi2 = make_float2(sphi, sphi);
    const float m2b = __fmul_rn(-2.0f, t.beta);
    const float2 m2b2 = make_float2(m2b, m2b);
    auto proj2 = [&](float ta, float tb) {
        float2 sn, cn;
        __sincosf(ta, &sn.x, &cn.x);
        __sincosf(tb, &sn.y, &cn.y);
        return __ffma2_rn(sn, sphi2, __fmul2_rn(cn, cphi2));
    };
    for (uint32_t u = warp; u < nzb * nseg; u += nwarps) {
        const uint32_t zb = u / nseg, y_lo = (u - zb * nseg) * seg, y_hi = min(g.ly, y_lo + seg);
        if (y_lo >= y_hi) continue;
        const uint32_t z = min(2 * (zb * groups + sub), g.lz - 2), z2 = z + 2 == g.lz ? 0u : z + 2;
        const float2 jx = make_float2(s.jxy[z], s.jxy[z + 1]), jzz = make_float2(s.jz[z], s.jz[z + 1]);
        /* z is even: the site (x, y) has colour (x + y) & 1 on planes z and z + 2, the other on z + 1 */
        uint32_t col = ((xl + y_lo) & 1u) ? g.stride1 : 0u;
        uint32_t o = y_lo * hx + (xl >> 1);
        const float *p0 = s.th + z * ph, *p1 = p0 + ph, *p2 = s.th + z2 * ph;
        float2 r = proj2(p0[col + o], p1[g.stride1 - col + o]);
        uint32_t idx = z * g.plane + y_lo * g.lx + xl;
        uint32_t k[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll kUnroll
        for (uint32_t y = y_lo; y < y_hi; ++y) {
            const uint32_t on = y + 1 == g.ly ? (xl >> 1) : o + hx, coln = g.stride1 - col;
            const float2 ry = proj2(p0[coln + on], p1[col + on]);
            float sn, cn;
            __sincosf(p2[col + o], &sn, &cn);
            const float2 rz = make_float2(r.y, wolff_projection(cn, sn, cphi, sphi));
            const float2 rx = make_float2(__shfl_sync(0xffffffffu, r.x, xsrc), __shfl_sync(0xffffffffu, r.y, xsrc));
            const slsf_u32x4 b0 = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_BOND, 0, idx);
            const slsf_u32x4 b1 = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_BOND, 0, idx + g.plane);
            const float2 jr = __fmul2_rn(jx, r);
            uint32_t w[6];
            wolff_bond_words(__fmul2_rn(jr, rx), m2b2, b0.x, b1.x, w[0], w[3]);
            wolff_bond_words(__fmul2_rn(jr, ry), m2b2, b0.y, b1.y, w[1], w[4]);
            wolff_bond_words(__fmul2_rn(__fmul2_rn(jzz, r), rz), m2b2, b0.z, b1.z, w[2], w[5]);
#pragma unroll
            for (int j = 0; j < 6; ++j) k[j] = lane == y - y_lo ? w[j] : k[j];
            r = ry;
            col = coln;
            o = on;
            idx += g.lx;
        }
        if (lane < y_hi - y_lo)
            for (uint32_t q = 0; q < groups && zb * groups + q < (g.lz >> 1); ++q) {
                const uint32_t row = row_word(g, y_lo + lane, 2 * (zb * groups + q)), sh = q * g.lx;
                s.bx[row] = (k[0] >> sh) & g.xmask;
                s.by[row] = (k[1] >> sh) & g.xmask;
                s.bz[row] = (k[2] >> sh) & g.xmask;
                s.bx[row + g.ly] = (k[3] >> sh) & g.xmask;
                s.by[row + g.ly] = (k[4] >> sh) & g.xmask;
                s.bz[row + g.ly] = (k[5] >> sh) & g.xmask;
            }
    }
}

/* One Wolff update (src/updates.rs:551-620); returns the thread's share of the cluster size. */
template <int kUnroll>
__device__ __forceinline__ uint32_t wolff_update(const TaskView& t, const Geo& g, Smem& s, uint64_t counter) {
    const slsf_u32x4 pick = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_PICK, 0, 0);
    const float phi = slsf_angle_from_word(pick.x);
    const uint32_t x0 = slsf_range(pick.y, g.lx), y0 = slsf_range(pick.z, g.ly), z0 = slsf_range(pick.w, g.lz);
    float sphi, cphi;
    __sincosf(phi, &sphi, &cphi);
    wolff_bonds<kUnroll>(t, g, s, counter, cphi, sphi);
    const uint32_t seed_row = row_word(g, y0, z0);
    for (uint32_t r = threadIdx.x; r < g.rows; r += blockDim.x) s.cl[r] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) s.cl[seed_row] = close_word(1u << x0, s.bx[seed_row], g.lx, true);
    __syncthreads();
    SLSF_PHASE(2);

    /* Grow the seed's component; every pass that goes on adds at least one
     * site, so the count is bounded by V (or the context's loop limit). */
    const uint32_t passes = grow(g, s, (t.loop_limit ? min(t.loop_limit, g.volume) : g.volume) + 1);
    if (passes == 0 && threadIdx.x == 0) atomicOr(&t.stats[kStatError], kErrGrowthLimit);
    SLSF_PHASE(3);
    SLSF_PHASE_COUNT(6, passes);
    SLSF_PHASE_COUNT(7, 1);

    /* Reflect the cluster (src/updates.rs:602-617) and count it. */
    uint32_t members = 0;
    for (uint32_t r = threadIdx.x; r < g.rows; r += blockDim.x) members += __popc(s.cl[r]);
    if (g.lx % 4 == 0) {
        /* four consecutive sites of a row (a pair of each colour) per thread
         * and step; a row's pairs are swapped between the colours by its parity */
        const uint32_t nq = g.lx >> 2;
        for (uint32_t i = threadIdx.x; i < (g.volume >> 2); i += blockDim.x) {
            const uint32_t r = slsf_fastdiv_div(i, g.div_nq), q = i - r * nq;
            const uint32_t z = slsf_fastdiv_div(r, g.div_ly), y = r - z * g.ly;
            const uint32_t m = s.cl[row_word(g, y, z)] >> (4 * q) & 15u;
            if (!m) continue;
            const uint32_t p = (y + z) & 1u; /* colour of the even-x sites */
            float2* even = reinterpret_cast<float2*>(s.th + p * g.stride1 + 2 * i);
            float2* odd = reinterpret_cast<float2*>(s.th + (p ^ 1u) * g.stride1 + 2 * i);
            float2 e = *even, o = *odd;
            const float ex = slsf_reflect(e.x, phi), ox = slsf_reflect(o.x, phi);
            const float ey = slsf_reflect(e.y, phi), oy = slsf_reflect(o.y, phi);
            e.x = (m & 1u) ? ex : e.x;
            o.x = (m & 2u) ? ox : o.x;
            e.y = (m & 4u) ? ey : e.y;
            o.y = (m & 8u) ? oy : o.y;
            *even = e;
            *odd = o;
        }
    } else {
        /* rows of 2 mod 4: a pair of neighbours, one site of each colour (a site
         * per thread took 53 us per sweep of a few 26^3 where this takes 51, and
         * 95 of 30^3 on 256 threads for 87) */
        const uint32_t hx = g.lx >> 1;
        for (uint32_t i = threadIdx.x; i < g.half; i += blockDim.x) {
            const uint32_t r = slsf_fastdiv_div(i, g.div_hx), k = i - r * hx;
            const uint32_t z = slsf_fastdiv_div(r, g.div_ly), y = r - z * g.ly;
            const uint32_t m = s.cl[row_word(g, y, z)] >> (2 * k) & 3u;
            if (!m) continue;
            const uint32_t p = (y + z) & 1u;
            float* even = s.th + p * g.stride1 + i;
            float* odd = s.th + (p ^ 1u) * g.stride1 + i;
            const float e = *even, o = *odd, e_new = slsf_reflect(e, phi), o_new = slsf_reflect(o, phi);
            *even = (m & 1u) ? e_new : e;
            *odd = (m & 2u) ? o_new : o;
        }
    }
    __syncthreads();
    SLSF_PHASE(4);
    return members;
}

/* Adds a per-thread count of the whole item to a shared total. */
__device__ __forceinline__ void item_total(unsigned long long v, unsigned long long* total) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31u) == 0 && v) atomicAdd(total, v);
}

/* (cos, sin) of the site (x, y, z) of the resident state. */
__device__ __forceinline__ float2 trig_at(const Geo& g, const Smem& s, uint32_t x, uint32_t y, uint32_t z) {
    float sn, cn;
    __sincosf(s.th[slot(g, x + g.lx * (y + g.ly * z), (x + y + z) & 1u)], &sn, &cn);
    return make_float2(cn, sn);
}

/* FP64 sum over the warp's lanes (the same shuffle tree everywhere). */
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

/* Correlation functions of the resident state (measure_theta_correlations_with_scratch,
 * src/observables.rs:165-270), measured between sweeps and added into row
 * count / binsize of the task's correlation bins in ThetaModel::measure's
 * order (C_x, C_y, C_xy, C_xy(z, r), C_z).  Per layer z a warp takes the x
 * lines (lane = x; partners at x + r by shuffle within the row) and the y
 * lines (lane = x; a register window of 8 partners slides along y); per row
 * y a warp takes the z lines the same way along z.  Products are FP32 fused
 * multiply-adds summed per lane over one line length (<= 32), lanes and
 * layers in FP64 in a fixed order.  Scratch (shared): sx, sy [L_z][R] and the
 * per-row z sums [L_y][R_z]. */
__device__ __noinline__ void corr_measure(const ResidentCorr& c, const Geo& g, const Smem& s) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t R = c.rxy, Rz = c.rz, lx = g.lx, ly = g.ly, lz = g.lz;
    double* sx = s.corr;
    double* sy = sx + lz * R;
    double* szr = sy + lz * R;
    const bool xv = lane < lx;
    const uint32_t x = xv ? lane : 0u;
    for (uint32_t u = warp; u < lz + ly; u += nwarps) {
        if (u < lz) {
            const uint32_t z = u;
            for (uint32_t r0 = 1; r0 <= R; r0 += 8) {
                /* x lines: the partner of x at lag r is lane (x + r) mod L_x of the row */
                uint32_t src[8];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) src[j] = (x + r0 + j) % lx;
                float ax[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                float ay[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                /* y lines: w[j] = partner (x, k + r0 + j) of the current k */
                float2 w[8];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) w[j] = trig_at(g, s, x, (r0 + j) % ly, z);
                uint32_t nxt = (r0 + 8) % ly; /* y of the partner entering the window after k */
                for (uint32_t k = 0; k < ly; ++k) {
                    float2 a = trig_at(g, s, x, k, z);
                    if (!xv) a = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) {
                        const float pc = __shfl_sync(0xffffffffu, a.x, src[j]);
                        const float ps = __shfl_sync(0xffffffffu, a.y, src[j]);
                        ax[j] = __fmaf_rn(a.y, ps, __fmaf_rn(a.x, pc, ax[j]));
                        ay[j] = __fmaf_rn(a.y, w[j].y, __fmaf_rn(a.x, w[j].x, ay[j]));
                    }
#pragma unroll
                    for (uint32_t j = 0; j + 1 < 8; ++j) w[j] = w[j + 1];
                    w[7] = trig_at(g, s, x, nxt, z);
                    nxt = nxt + 1 == ly ? 0u : nxt + 1;
                }
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const double vx = warp_total((double)ax[j]), vy = warp_total((double)ay[j]);
                    if (lane == 0 && r0 + j <= R) {
                        sx[z * R + r0 + j - 1] = vx;
                        sy[z * R + r0 + j - 1] = vy;
                    }
                }
            }
        } else {
            const uint32_t y = u - lz;
            for (uint32_t r0 = 1; r0 <= Rz; r0 += 8) {
                /* z lines of row y: w[j] = partner (x, y, k + r0 + j) */
                float az[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                float2 w[8];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) w[j] = trig_at(g, s, x, y, (r0 + j) % lz);
                uint32_t nxt = (r0 + 8) % lz;
                for (uint32_t k = 0; k < lz; ++k) {
                    float2 a = trig_at(g, s, x, y, k);
                    if (!xv) a = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) az[j] = __fmaf_rn(a.y, w[j].y, __fmaf_rn(a.x, w[j].x, az[j]));
#pragma unroll
                    for (uint32_t j = 0; j + 1 < 8; ++j) w[j] = w[j + 1];
                    w[7] = trig_at(g, s, x, y, nxt);
                    nxt = nxt + 1 == lz ? 0u : nxt + 1;
                }
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const double v = warp_total((double)az[j]);
                    if (lane == 0 && r0 + j <= Rz) szr[y * Rz + r0 + j - 1] = v;
                }
            }
        }
    }
    __shared__ unsigned long long s_row;
    if (threadIdx.x == 0) s_row = *c.count / c.binsize;
    __syncthreads();
    if (s_row < c.n_bins) {
        const uint32_t nv = 3 * R + lz * R + Rz;
        double* bin = c.bins + s_row * nv;
        const double volume = (double)g.volume, area = (double)g.plane;
        for (uint32_t j = threadIdx.x; j < lz * R; j += blockDim.x) bin[3 * R + j] += (sx[j] + sy[j]) / (2.0 * area);
        for (uint32_t r = threadIdx.x; r < R; r += blockDim.x) {
            double a = 0.0, b = 0.0;
            for (uint32_t z = 0; z < lz; ++z) {
                a += sx[z * R + r];
                b += sy[z * R + r];
            }
            const double cx = a / volume, cy = b / volume;
            bin[r] += cx;
            bin[R + r] += cy;
            bin[2 * R + r] += (cx + cy) / 2.0;
        }
        for (uint32_t r = threadIdx.x; r < Rz; r += blockDim.x) {
            double a = 0.0;
            for (uint32_t y = 0; y < ly; ++y) a += szr[y * Rz + r];
            bin[3 * R + lz * R + r] += a / volume;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) *c.count += 1;
}

/* Fused observables of the resident state (src/observables.rs:99-141): mx,
 * my, cos xyz, sin xyz; FP64 sums of the FP32 bond terms, block total valid
 * in thread 0. */
__device__ __forceinline__ void measure(const Geo& g, const Smem& s, double (&acc)[8], double* red) {
    const uint32_t lane = threadIdx.x & 31u;
    double f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t i0 = (threadIdx.x & ~31u); i0 < g.volume; i0 += blockDim.x) {
        const uint32_t idx = i0 + lane;
        const bool valid = idx < g.volume;
        const uint32_t ii = valid ? idx : 0;
        const Coords c = coords_of(g, ii);
        uint32_t xp, yp, zp;
        forward_neighbours(g, ii, c, xp, yp, zp);
        float si, ci, sx, cx, sy, cy, sz, cz;
        __sincosf(site_theta(g, s, ii, c), &si, &ci);
        if (g.lx_tiles_warp) {
            const uint32_t src = xp_lane(lane, g.lx);
            sx = __shfl_sync(0xffffffffu, si, src);
            cx = __shfl_sync(0xffffffffu, ci, src);
        } else {
            const Coords cxp = {c.x + 1 == g.lx ? 0 : c.x + 1, c.y, c.z, c.row};
            __sincosf(site_theta(g, s, xp, cxp), &sx, &cx);
        }
        const Coords cyp = {c.x, c.y + 1 == g.ly ? 0 : c.y + 1, c.z, 0};
        const Coords czp = {c.x, c.y, c.z + 1 == g.lz ? 0 : c.z + 1, 0};
        __sincosf(site_theta(g, s, yp, cyp), &sy, &cy);
        __sincosf(site_theta(g, s, zp, czp), &sz, &cz);
        if (!valid) continue;
        const float jx = s.jxy[c.z], jzz = s.jz[c.z];
        f[0] += ci;
        f[1] += si;
        f[2] += bond_cos(jx, ci, si, cx, sx);
        f[3] += bond_cos(jx, ci, si, cy, sy);
        f[4] += bond_cos(jzz, ci, si, cz, sz);
        f[5] += bond_sin(jx, ci, si, cx, sx);
        f[6] += bond_sin(jx, ci, si, cy, sy);
        f[7] += bond_sin(jzz, ci, si, cz, sz);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = f[k];
    block_sum<8>(acc, red);
}


constexpr int kLongRuns = 4; /* kUnroll of 512-thread CTAs (launch_resident) */

/* kCorr: with fused correlations; kUnroll: rows unrolled in the bond activation. */
template <bool kCorr, int kMaxThreads, int kUnroll>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_resident(const TaskView* __restrict__ views, uint32_t n, uint32_t n_sweeps, unsigned int* __restrict__ queue,
               uint32_t max_volume, uint32_t max_rows, uint32_t max_lz, unsigned long long* __restrict__ counters,
               const ResidentCorr* __restrict__ corr, TaskView one) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[8 * 32];
    __shared__ double bin_acc[kBinCols];
    __shared__ uint32_t s_item;
    /* 64 bits: an item's counts run over all of its sweeps (2^32 accepted sites are 131,072 sweeps at 32^3) */
    __shared__ unsigned long long s_cluster;
    __shared__ unsigned long long s_accepted;
    for (bool first = true;; first = false) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = queue ? atomicAdd(queue, 1u) : (first ? 0u : n);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n) return;
        TaskView t = views ? views[item] : one; /* one task by value: no view in device memory, no queue */
        if (counters) { /* a replayed launch: the counters live in their own array */
            t.metro_sweeps = counters[2 * item];
            t.wolff_done = counters[2 * item + 1];
        }
        const Geo g = make_geo(t);
        Smem s = carve(smem_raw, max_volume, max_rows, max_lz);
        if (threadIdx.x == 0) {
            s_cluster = 0;
            s_accepted = 0;
        }
        load_state(t, g, s);
        __syncthreads();
#ifdef SLSF_PHASE_TIMING
        if (threadIdx.x == 0) s_phase_mark = clock64();
#endif
        const uint32_t sweeps = t.sweeps ? t.sweeps : n_sweeps;
        unsigned long long accepted = 0, cluster_sites = 0;
        int64_t bin_cur = -1;
        /* ThetaModel::measure after every sweep past thermalization: the state
         * after sweep k is measured inside sweep k+1's colour-0 half-sweep,
         * the launch's last state by the measurement pass below. */
        const bool measuring = t.n_bins > 0;
        for (uint32_t sw = 0; sw < sweeps; ++sw) {
            const uint64_t sweep = t.metro_sweeps + sw;
            if (!t.wolff_only) {
                double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (measuring && sw > 0 && sweep > t.thermalization) {
                    accepted += sweep_colour<true>(t, g, s, sweep, 0, acc);
                    double tot[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) tot[k] = acc[k];
                    block_sum<8>(tot, red);
                    if (threadIdx.x == 0) bin_measurement(t, g.volume, sweep, tot, bin_acc, bin_cur);
                } else {
                    accepted += sweep_colour<false>(t, g, s, sweep, 0, acc);
                }
                __syncthreads();
                SLSF_PHASE(0);
                accepted += sweep_colour<false>(t, g, s, sweep, 1, acc);
                __syncthreads();
                SLSF_PHASE(1);
            }
            for (uint32_t k = 0; k < t.wolff_steps; ++k)
                cluster_sites += wolff_update<kUnroll>(t, g, s, t.wolff_done + (uint64_t)sw * t.wolff_steps + k);
            /* ThetaModel::measure's correlations of the state after this sweep:
             * measurement m = sweep - thermalization, every corr_interval-th */
            if constexpr (kCorr) {
                const ResidentCorr& c = corr[item];
                if (c.bins && sweep >= t.thermalization && (sweep - t.thermalization) % c.interval == 0) {
                    __syncthreads();
                    corr_measure(c, g, s);
                    __syncthreads();
                }
            }
        }
        const uint64_t last = t.metro_sweeps + sweeps;
        /* the counters advance on the device, so that a replayed launch
         * (slsf_batch_open / slsf_batch_step) continues the streams; every
         * thread read them before the first barrier of the item */
        if (counters && threadIdx.x == 0) {
            counters[2 * item] = last;
            counters[2 * item + 1] = t.wolff_done + (uint64_t)sweeps * t.wolff_steps;
        }
        if (measuring && sweeps > 0 && last > t.thermalization) {
            double acc[8];
            measure(g, s, acc, red);
            SLSF_PHASE(5);
            if (threadIdx.x == 0) bin_measurement(t, g.volume, last, acc, bin_acc, bin_cur);
        }
        if (threadIdx.x == 0) flush_bin(t, bin_acc, bin_cur);
        item_total(accepted, &s_accepted);
        item_total(cluster_sites, &s_cluster);
        __syncthreads();
        store_state(t, g, s);
        if (threadIdx.x == 0 && views) {
            atomicAdd(&t.stats[kStatAccepted], s_accepted);
            atomicAdd(&t.stats[kStatClusterSites], s_cluster);
            atomicAdd(&t.stats[kStatClusters], (unsigned long long)sweeps * t.wolff_steps);
        } else if (threadIdx.x == 0) { /* the call's counters, to the host (t.stats is pinned memory) */
            t.stats[kStatAccepted] = s_accepted;
            t.stats[kStatClusterSites] = s_cluster;
            t.stats[kStatClusters] = (unsigned long long)sweeps * t.wolff_steps;
        }
    }
}

size_t smem_bytes(uint32_t max_volume, uint32_t max_rows, uint32_t max_lz, uint32_t corr_doubles = 0) {
    return 4ull * (max_volume + 2 * kPad) + 16ull * max_rows + 8ull * max_lz + 8ull * corr_doubles;
}

/* Compute capability 10.0 gives a block 227 KB; the kernel's static arrays need room in it. */
constexpr size_t kMaxDynamicSmem = 227 * 1024 - 4096;

/* Lets a kernel be launched with `smem` bytes: its limit goes to the device's
 * at once, since a limit as low as one launch needs would refuse the larger
 * launch that another thread, with a context of its own, is about to make. */
template <typename K>
cudaError_t allow_smem(K kernel, size_t smem) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(smem, kMaxDynamicSmem));
}

template <bool kCorr, int kMaxThreads, int kUnroll>
cudaError_t launch_resident_t(const TaskView* views_dev, uint32_t n, uint32_t n_sweeps, unsigned int* queue,
                              int device, cudaStream_t s, uint32_t max_volume, uint32_t max_rows, uint32_t max_lz,
                              uint32_t threads, unsigned long long* counters, const ResidentCorr* corr,
                              uint32_t corr_doubles) {
    const size_t smem = smem_bytes(max_volume, max_rows, max_lz, corr_doubles);
    const TaskView none = {};
    cudaError_t e = allow_smem(k_resident<kCorr, kMaxThreads, kUnroll>, smem);
    if (e != cudaSuccess) return e;
    int sms = 0, per_sm = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resident<kCorr, kMaxThreads, kUnroll>, (int)threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const uint32_t grid = std::min<uint32_t>(n, (uint32_t)(sms * per_sm));
    k_resident<kCorr, kMaxThreads, kUnroll><<<grid, threads, smem, s>>>(views_dev, n, n_sweeps, queue, max_volume, max_rows, max_lz,
                                                  counters, corr, none);
    return cudaGetLastError();
}

}  // namespace

bool resident_supports(uint32_t lx, uint32_t ly, uint32_t lz) {
    /* Row words hold L_x <= 32 bits; the colour-split layout needs even
     * dimensions (L_x = 2 mod 4 copies the state site by site). */
    if (lx > kMaxRowBits || lx < 4 || lx % 2 || ly < 2 || ly % 2 || lz < 2 || lz % 2) return false;
    const uint64_t v = (uint64_t)lx * ly * lz;
    return smem_bytes((uint32_t)v, ly * lz, lz) <= kMaxDynamicSmem;
}

cudaError_t launch_resident_one(const TaskView& t, uint32_t n_sweeps, uint32_t threads, cudaStream_t s) {
    const uint32_t volume = t.lx * t.ly * t.lz;
    const size_t smem = smem_bytes(volume, t.ly * t.lz, t.lz);
    cudaError_t e = allow_smem(k_resident<false, 512, 1>, smem);
    if (e != cudaSuccess) return e;
    TaskView v = t;
    v.sweeps = n_sweeps;
    k_resident<false, 512, 1><<<1, threads, smem, s>>>(nullptr, 1, n_sweeps, nullptr, volume, t.ly * t.lz, t.lz, nullptr,
                                                    nullptr, v);
    return cudaGetLastError();
}

uint32_t resident_corr_doubles(uint32_t ly, uint32_t lz, uint32_t rxy, uint32_t rz) {
    return (rxy || rz) ? 2 * lz * rxy + ly * rz : 0;
}

cudaError_t launch_resident(const TaskView* views_dev, uint32_t n, uint32_t n_sweeps, unsigned int* queue,
                            int device, cudaStream_t s, uint32_t max_volume, uint32_t max_rows, uint32_t max_lz,
                            uint32_t threads, unsigned long long* counters, const ResidentCorr* corr_dev,
                            uint32_t corr_doubles) {
    if (threads < 32 || threads > (uint32_t)kBThreads || threads % 32) return cudaErrorInvalidConfiguration;
    /* lattices that take 512 threads have long bond runs and an SM to
     * themselves: four rows unrolled give 7.34e10 site-updates/s over 1184
     * replicas of 32^3 for 7.20e10 (22^3 to 30^3 and 12x50x50 2 to 3 % more);
     * smaller ones, whose CTAs share an SM's instruction cache, lose by it
     *
     * the fused correlation measurement is compiled into its own instances, so
     * groups without it run the kernel unchanged; CTAs of up to 512 threads
     * have 128 registers a thread (the patch walk and its compensated sums
     * need about 120), larger ones 64 and spill: 6.67e10 against 5.8e10
     * site-updates/s at L = 32 */
    if (corr_dev && corr_doubles)
        return threads > 512 ? launch_resident_t<true, kBThreads, 1>(views_dev, n, n_sweeps, queue, device, s, max_volume,
                                                                  max_rows, max_lz, threads, counters, corr_dev,
                                                                  corr_doubles)
                             : launch_resident_t<true, 512, 1>(views_dev, n, n_sweeps, queue, device, s, max_volume,
                                                            max_rows, max_lz, threads, counters, corr_dev,
                                                            corr_doubles);
    const auto launch = threads > 512    ? launch_resident_t<false, kBThreads, 1>
                        : threads == 512 ? launch_resident_t<false, 512, kLongRuns>
                                         : launch_resident_t<false, 512, 1>;
    return launch(views_dev, n, n_sweeps, queue, device, s, max_volume, max_rows, max_lz, threads, counters, nullptr, 0);
}

}  // namespace slsf

#ifdef SLSF_PHASE_TIMING
extern "C" int slsf_debug_resident_phase_cycles(unsigned long long out[8], int reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, slsf::g_res_phase_cycles, sizeof(unsigned long long) * 8);
    if (e == cudaSuccess && reset) {
        const unsigned long long zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        e = cudaMemcpyToSymbol(slsf::g_res_phase_cycles, zero, sizeof(zero));
    }
    return e == cudaSuccess ? 0 : 1;
}
#endif
