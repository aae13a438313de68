/*
 * Wolff update of a lattice in global memory on bit-packed bonds: the bond
 * activation of a warp's run of rows, the reflection of four sites and the
 * closure of rows of up to 64 sites, for kernel_wolff_bits.cu (one lattice)
 * and kernel_stream.cu (many replicas, persistent).  Bit x mod 32 of word
 * x / 32 of a row is site x; a row takes ceil(L_x / 32) words.
 */
#ifndef SLSF_WOLFF_GLOBAL_CUH
#define SLSF_WOLFF_GLOBAL_CUH

#include "bitgrow.cuh"
#include "fastdiv.h"
#include "xy_device.cuh"

namespace slsf {

/* Bond activation.  A warp owns word w (lane = bit = x - 32 w; lanes past the
 * row keep no bits) of the plane pair z, z + 1 for a run of up to 32 rows and
 * walks it along y, so the projections of the +y row are the next row's own
 * and plane z's +z partner is plane z + 1's site: three sincos for its two
 * sites, whose arithmetic is packed and whose Philox blocks share a key
 * schedule.  (The earlier walk of one plane took 186 instructions per site and
 * 133 us at L = 256, this one 100 and 84.)  Lane j keeps the words of the
 * run's row j and writes them at its end.  With an odd L_z the last pair's second plane is plane 0,
 * computed and not kept. */
struct BitPlanes {
    uint32_t *bx, *by, *bz, *cl; /* [rows][words] */
};

/* (theta is not __restrict__: the persistent kernel changes the angles between its phases.  kRows: rows in flight.) */
template <int kRows>
__device__ __forceinline__ void bond_run(const float* theta, const float* __restrict__ jxy,
                                         const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz,
                                         float minus_two_beta, float phi, uint64_t seed, uint64_t counter,
                                         const BitPlanes& wb, uint32_t run, uint32_t wid,
                                         uint8_t* __restrict__ bond_bytes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t words = (lx + 31u) >> 5, nrun = (ly + run - 1) / run;
    const uint32_t w = wid % words, rest = wid / words;
    const uint32_t z = 2u * (rest / nrun), y_lo = (rest % nrun) * run;
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
#pragma unroll kRows
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

/* Reflects the cluster's sites among four consecutive ones of a row, kN quads
 * of the lattice per thread a distance `step` apart with their loads in flight
 * together (one 16-byte access each when L_x is a multiple of 4 and the angles
 * are aligned: `wide`), with an optional byte mask; returns their number. */
template <int kN>
__device__ __forceinline__ uint32_t flip_quads(float* theta, uint32_t lx, uint32_t rows, uint32_t q0, uint32_t step,
                                               const slsf_fastdiv& quads, const uint32_t* cl, float phi,
                                               uint8_t* __restrict__ cluster_out, bool wide) {
    uint32_t m[kN], n = 0;
    size_t at[kN];
    float4 v[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
        const uint32_t q = q0 + j * step, row = slsf_fastdiv_div(q, quads), x = 4u * (q - row * quads.d);
        at[j] = (size_t)row * lx + x;
        m[j] = q < quads.d * rows ? (__ldcg(&cl[row * ((lx + 31u) >> 5) + (x >> 5)]) >> (x & 31u)) & 0xfu : 0u;
        if (cluster_out && q < quads.d * rows)
            for (uint32_t k = 0; k < min(4u, lx - x); ++k) cluster_out[at[j] + k] = (uint8_t)(m[j] >> k & 1u);
    }
    if (wide) {
#pragma unroll
        for (int j = 0; j < kN; ++j)
            if (m[j]) v[j] = *reinterpret_cast<const float4*>(theta + at[j]);
    }
#pragma unroll
    for (int j = 0; j < kN; ++j) {
        n += __popc(m[j]);
        if (!m[j]) continue;
        if (wide) {
            v[j].x = m[j] & 1u ? slsf_reflect(v[j].x, phi) : v[j].x;
            v[j].y = m[j] & 2u ? slsf_reflect(v[j].y, phi) : v[j].y;
            v[j].z = m[j] & 4u ? slsf_reflect(v[j].z, phi) : v[j].z;
            v[j].w = m[j] & 8u ? slsf_reflect(v[j].w, phi) : v[j].w;
            *reinterpret_cast<float4*>(theta + at[j]) = v[j];
        } else {
            for (uint32_t k = 0; k < 4; ++k)
                if (m[j] >> k & 1u) theta[at[j] + k] = slsf_reflect(theta[at[j] + k], phi);
        }
    }
    return n;
}

/* Closure of a periodic row of up to 64 sites along x (close_word); kWhole: a
 * row of exactly one or two words, whose reversal and carry need no shifts. */
template <bool kWhole>
__device__ __forceinline__ uint64_t carry_up64(uint64_t c, uint64_t b, uint32_t lx) {
    uint64_t s = b + (c & b);
    c |= kWhole ? (uint64_t)(s < b) : s >> lx;
    s = b + (c & b);
    return (s ^ b) | c;
}

template <bool kWhole>
__device__ __forceinline__ uint64_t close_row(uint64_t c, uint64_t b, uint32_t lx) {
    if (kWhole) {
        const uint64_t bl = (b << 1) | (b >> 63);
        return carry_up64<true>(c, b, 64) | __brevll(carry_up64<true>(__brevll(c), __brevll(bl), 64));
    }
    const uint64_t mask = ~0ull >> (64 - lx), bl = ((b << 1) | (b >> (lx - 1))) & mask;
    const uint32_t sh = 64 - lx;
    return (carry_up64<false>(c, b, lx) | (__brevll(carry_up64<false>(__brevll(c) >> sh, __brevll(bl) >> sh, lx)) >> sh)) & mask;
}

template <bool kWhole>
__device__ __forceinline__ uint32_t close_row(uint32_t c, uint32_t b, uint32_t lx) {
    return close_word(c, b, kWhole ? 32u : lx, true);
}

}  // namespace slsf

#endif /* SLSF_WOLFF_GLOBAL_CUH */
