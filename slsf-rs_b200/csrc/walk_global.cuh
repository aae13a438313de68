/*
 * Walks over one lattice in global memory, L_x a multiple of 4: the work of
 * one thread of kernel_walk.cu (one lattice per launch) and kernel_stream.cu
 * (many replicas, persistent).
 *
 * A thread reads the four sites x = 4 q .. 4 q + 3 of a row with one 16-byte
 * load (the angles are one 256-byte aligned array and L_x is a multiple of 4)
 * and gets a pair of each colour.  A colour's update writes only that colour;
 * its 16-byte stores put back the other colour's words as they were, which no
 * thread changes meanwhile.
 */
#ifndef SLSF_WALK_GLOBAL_CUH
#define SLSF_WALK_GLOBAL_CUH

#include "engine.h"
#include "walk.cuh"
#include "xy_device.cuh"

namespace slsf {

/* Bin row of the state after `done` sweeps, NULL if it is not measured or kept. */
__device__ __forceinline__ double* bin_row_of(const TaskView& t, uint64_t done) {
    if (t.n_bins == 0 || done <= t.thermalization) return nullptr;
    const uint64_t b = (done - t.thermalization - 1) / t.binsize;
    return b < t.n_bins ? t.bins + b * kBinCols : nullptr;
}

/* Adds the measured values of totals `tot` to a bin row in the batched
 * kernels' column order (ThetaModel::measure's stream, src/model.rs:406-409). */
__device__ __forceinline__ void add_to_bin(const TaskView& t, const double (&tot)[8], double* bin_row) {
    const double v = (double)(t.lx * t.ly * t.lz);
    const double e = -(tot[2] + tot[3] + tot[4]) / v;
    const double vals[kBinCols] = {e,      e * e,  (tot[0] * tot[0] + tot[1] * tot[1]) / (v * v),
                                   tot[2], tot[3], tot[4],
                                   tot[5], tot[6], tot[7],
                                   tot[5] * tot[5], tot[6] * tot[6], tot[7] * tot[7]};
    for (int q = 0; q < kBinCols; ++q) bin_row[q] += vals[q];
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

/* Units (threads' patches) of a replica. */
__host__ __device__ inline uint32_t walk_units(const TaskView& t, uint32_t seglen) {
    return (t.lx >> 2) * (t.ly >> 1) * ((t.lz + seglen - 1) / seglen);
}

/* One colour of unit `unit`'s patch; returns the accepted sites and, with
 * kMeasure, adds the terms of the state before the update to sums. */
template <bool kMeasure>
__device__ __forceinline__ uint32_t walk_colour(const TaskView& t, uint64_t sweep, uint32_t colour, uint32_t seglen,
                                                uint32_t unit_index, WalkSums* sums) {
    const uint32_t lx = t.lx, plane = lx * t.ly;
    uint32_t accepted = 0;
    Patch pt;
    if (!patch_of(t, unit_index, seglen, pt)) return 0;
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
    Sum2* sum = kMeasure ? sums->run : nullptr;
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
    uint32_t z = pt.z_lo + par_lo;
    if (par_lo) step(pt.z_lo, std::true_type());
    for (; z + 1 < pt.z_hi; z += 2) {
        step(z, std::false_type());
        step(z + 1, std::true_type());
        if (kMeasure) sums->flush();
    }
    /* planes that no pair has flushed: the last, or an only one */
    const bool open = z < pt.z_hi || pt.z_hi - pt.z_lo == 1;
    if (z < pt.z_hi) step(z, std::false_type());
    if (kMeasure && open) sums->flush();
    return accepted;
}

/* J cos and J sin of the bonds a -> b of two sites. */
__device__ __forceinline__ void add_bond2(Sum2& ac, Sum2& as, float j, const Trig2& a, const Trig2& b) {
    ac.add(__fmul2_rn(dup2(j), __ffma2_rn(a.c, b.c, __fmul2_rn(a.s, b.s))));
    as.add(__fmul2_rn(dup2(j), __ffma2_rn(a.s, b.c, __fmul2_rn(neg2(a.c), b.s))));
}

/* The observables' terms of unit `unit`'s patch, added to sums. */
__device__ __forceinline__ void walk_measure(const TaskView& t, uint32_t seglen, uint32_t unit_index, WalkSums& sums) {
    const uint32_t lx = t.lx, plane = lx * t.ly;
    Patch pt;
    if (!patch_of(t, unit_index, seglen, pt)) return;
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
    Sum2* sum = sums.run;
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
        if (z & 1u) sums.flush();
    }
    if (pt.z_hi & 1u) sums.flush(); /* the last plane's terms */
}

}  // namespace slsf

#endif /* SLSF_WALK_GLOBAL_CUH */
