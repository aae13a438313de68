/*
 * Arithmetic of the walks: two sites per thread in packed FP32 instructions
 * (two operations each).  Shared by the batched one-CTA kernel
 * (kernel_resident.cu, the replica in shared memory) and the kernels over
 * lattices in global memory (kernel_walk.cu).  Every operation rounds as its
 * scalar form in xy_device.cuh, so decisions, angles and measured terms are
 * bit-identical to the site-by-site kernels.
 */
#ifndef SLSF_WALK_CUH
#define SLSF_WALK_CUH

#include <type_traits>

#include "xy_device.cuh"

namespace slsf {

struct Trig2 {
    float2 c, s; /* cos and sin of two sites */
};

__device__ __forceinline__ Trig2 trig2(float2 th) {
    Trig2 t;
    __sincosf(th.x, &t.s.x, &t.c.x);
    __sincosf(th.y, &t.s.y, &t.c.y);
    return t;
}

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

/* FP64 sums of FP32 terms of two sites, a few planes of them gathered in FP32
 * first: a value and a remainder per site.  The value starts at a bias that
 * keeps it above every term's magnitude, so each addition's rounding error is
 * exactly x - (t - v) (Dekker's fast two-sum); the errors add up in the
 * remainder.  Before kWalkRun planes and one are over, the two are added to the
 * thread's FP64 sum and start anew.  Up to then the value stays below 2^6 times
 * the terms' bound and the remainder below 2^-14, which rounds only where small
 * terms have bits past 2^-38 of the bound: against FP64 sums of the same terms
 * 2^-52 of their total, 2^-47 where the layers' couplings spread over six decades
 * (value and remainder kept for a whole walk: 2^-41 there, at 64 planes a
 * thread).  Four packed FP32 instructions per two terms and three conversions
 * per run, 1 to 2 % of a sweep more than one run per walk; converting each term
 * takes eight cycles of the special-function pipe, which bound the measuring
 * half-sweep (41k of 136k cycles per sweep at L = 32 against 18k for the other
 * colour; 32k with one run per walk). */
constexpr int kWalkRun = 2;
constexpr float kWalkBias = 8.0f * (kWalkRun + 1); /* twice the terms, four a plane, of kWalkRun + 1 planes */
struct Sum2 {
    float2 v, r;
    __device__ __forceinline__ void start(float bias) {
        v = make_float2(bias, bias);
        r = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void add(float2 x) {
        const float2 minus = make_float2(-1.0f, -1.0f);
        const float2 t = __fadd2_rn(v, x);
        r = __fadd2_rn(r, __ffma2_rn(__ffma2_rn(v, minus, t), minus, x));
        v = t;
    }
    /* The sum so far (v - bias is exact: v stays within a factor of two of the bias); starts anew. */
    __device__ __forceinline__ double take(float bias) {
        const double s = ((double)__fsub_rn(v.x, bias) + (double)__fsub_rn(v.y, bias)) + (double)__fadd_rn(r.x, r.y);
        start(bias);
        return s;
    }
};

/* Bound of the terms of sum k (mx, my, cos xyz, sin xyz): each direction's own
 * largest coupling, so that the weaker one's terms are not lost under the
 * other's bias. */
__device__ __forceinline__ float term_bound(float jxy_max, float jz_max, int k) {
    return k < 2 ? 1.0f : (k == 4 || k == 7 ? jz_max : jxy_max);
}

/* A walk's sums (mx, my, cos xyz, sin xyz): `flush` at the latest after kWalkRun
 * + 1 planes, `acc` holds them after it. */
struct WalkSums {
    Sum2 run[8];
    double acc[8];
    float jxy, jz;
    __device__ __forceinline__ float bias(int k) const { return kWalkBias * term_bound(jxy, jz, k); }
    __device__ __forceinline__ void start(float jxy_max, float jz_max) {
        jxy = jxy_max;
        jz = jz_max;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            run[k].start(bias(k));
            acc[k] = 0.0;
        }
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += run[k].take(bias(k));
    }
};

/* Adds J cos and J sin of the forward bonds i -> p and the backward bonds
 * m -> i of two sites i (bond_cos, bond_sin). */
__device__ __forceinline__ void add_bonds2(Sum2& ac, Sum2& as, float jp, float jm, const Trig2& i, const Trig2& n,
                                           const Trig2& p, const Trig2& m) {
    ac.add(__fmul2_rn(dup2(jp), __ffma2_rn(i.c, p.c, __fmul2_rn(i.s, p.s))));
    as.add(__fmul2_rn(dup2(jp), __ffma2_rn(i.s, p.c, __fmul2_rn(n.c, p.s))));
    ac.add(__fmul2_rn(dup2(jm), __ffma2_rn(m.c, i.c, __fmul2_rn(m.s, i.s))));
    as.add(__fmul2_rn(dup2(jm), __ffma2_rn(m.s, i.c, __fmul2_rn(m.c, n.s))));
}

/* field_from_pairs of two sites. */
__device__ __forceinline__ float2 field2(float jxy, float jzp, float jzm, float2 a01, float2 a23, float2 a4, float2 a5) {
    return __ffma2_rn(dup2(jzm), a5, __ffma2_rn(dup2(jzp), a4, __fmul2_rn(dup2(jxy), __fadd2_rn(a01, a23))));
}

/* metro_decide for the two sites of a Philox block; returns the number accepted. */
__device__ __forceinline__ uint32_t metro_pair(float2& th, const Trig2& own, float2 hx, float2 hy, float beta,
                                               float width, const slsf_u32x4& b) {
    const float2 up = make_float2((float)(b.x >> 8), (float)(b.z >> 8));
    /* 2 u - 1 with u = word >> 8 over 2^24 */
    const float2 d = __ffma2_rn(up, dup2(1.0f / 8388608.0f), dup2(-1.0f));
    const float2 t = __ffma2_rn(dup2(width), d, th);
    const float2 tn = make_float2(slsf_wrap_once(t.x), slsf_wrap_once(t.y));
    const Trig2 n = trig2(tn);
    const float2 dc = __fadd2_rn(own.c, neg2(n.c)), ds = __fadd2_rn(own.s, neg2(n.s));
    const float2 de = __ffma2_rn(dc, hx, __fmul2_rn(ds, hy));
    const float2 arg = __fmul2_rn(dup2(-beta), de);
    const bool a0 = (de.x <= 0.0f) | (slsf_u24f(b.y) < __expf(arg.x));
    const bool a1 = (de.y <= 0.0f) | (slsf_u24f(b.w) < __expf(arg.y));
    th.x = a0 ? tn.x : th.x;
    th.y = a1 ? tn.y : th.y;
    return (a0 ? 1u : 0u) + (a1 ? 1u : 0u);
}

/* The colour-c update of one row's pair of sites.  c: the other colour's trig
 * at the pair's compact indices; e: (cos, sin) of the x neighbour outside the
 * pair; dn, up, zm, zp: trig at -y, +y, -z, +z.  kOdd: the row's parity, whose
 * colour-c sites sit at x = 2 k + parity.  With kMeasure the terms of the
 * state before the update go to sum (mx, my, cos xyz, sin xyz). */
template <bool kMeasure, bool kOdd>
__device__ __forceinline__ uint32_t update_pair(float2& th, const Trig2& c, float2 e, const Trig2& dn, const Trig2& up,
                                                const Trig2& zm, const Trig2& zp, float jx, float jzp, float jzm,
                                                float beta, float width, const slsf_u32x4& b, Sum2* sum) {
    /* parity 0: +x is the other colour's same compact site, -x the previous; parity 1: -x the same, +x the next */
    Trig2 xp, xm;
    if (kOdd) {
        xp.c = make_float2(c.c.y, e.x);
        xp.s = make_float2(c.s.y, e.y);
        xm = c;
    } else {
        xp = c;
        xm.c = make_float2(e.x, c.c.x);
        xm.s = make_float2(e.y, c.s.x);
    }
    const Trig2 i = trig2(th);
    if (kMeasure) {
        /* the site and the other colour's site of the same index: each site once */
        sum[0].add(i.c);
        sum[1].add(i.s);
        sum[0].add(c.c);
        sum[1].add(c.s);
        Trig2 n; /* (-cos, -sin) of the site */
        n.c = neg2(i.c);
        n.s = neg2(i.s);
        add_bonds2(sum[2], sum[5], jx, jx, i, n, xp, xm);
        add_bonds2(sum[3], sum[6], jx, jx, i, n, up, dn);
        add_bonds2(sum[4], sum[7], jzp, jzm, i, n, zp, zm);
    }
    const float2 fx = field2(jx, jzp, jzm, __fadd2_rn(xp.c, xm.c), __fadd2_rn(up.c, dn.c), zp.c, zm.c);
    const float2 fy = field2(jx, jzp, jzm, __fadd2_rn(xp.s, xm.s), __fadd2_rn(up.s, dn.s), zp.s, zm.s);
    return metro_pair(th, i, fx, fy, beta, width, b);
}

}  // namespace slsf

#endif /* SLSF_WALK_CUH */
