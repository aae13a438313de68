/*
 * Bit-parallel closure of a Wolff cluster over active bonds: a row word along
 * x, shared by the batched one-CTA kernel (kernel_resident.cu) and the
 * large-lattice growth (kernel_wolff_bits.cu), and for the latter a block of
 * 32 x 32 words -- 32 rows along y by 32 planes along z, one 32-bit word of 32
 * sites along x per row -- closed in shared memory by warp scans.
 *
 * The cluster is the seed's connected component over the active bonds, the
 * set the reference's depth-first search collects (src/updates.rs:577-597)
 * when fed the same per-bond randoms.  Bits only ever get set, so every order
 * of the closure steps reaches the same fixed point.
 */
#ifndef SLSF_BITGROW_CUH
#define SLSF_BITGROW_CUH

#include <cuda_runtime.h>
#include <stdint.h>

namespace slsf {

constexpr uint32_t kGrowEdge = 32; /* rows per plane and planes per block */

/* Closure of the cluster bits c of one word along x through its bonds b (bit
 * j: bond j -- j+1).  periodic: the word is a whole row of lx <= 32 sites and
 * bit lx - 1 bonds to bit 0; otherwise it is a word of 32 sites, open at both
 * ends (bits crossing words enter between passes).  Bits above lx are zero.
 *
 * Adding the cluster's bits to the bond word carries through every run of
 * bonds: b + (c & b) differs from b in the bits from a seed to the site its
 * run ends on (except where a further seed lies, which c has).  The other
 * direction is the same on the reversed words.  About 20 instructions, against
 * 40 for doubling steps in both directions. */
__device__ __forceinline__ uint32_t carry_up(uint32_t c, uint32_t b, uint32_t lx, bool periodic) {
    uint32_t s = b + (c & b);
    if (periodic) {
        c |= lx == 32 ? (uint32_t)(s < b) : s >> lx; /* the carry out of the row enters site 0 */
        s = b + (c & b);
    }
    return (s ^ b) | c;
}

__device__ __forceinline__ uint32_t close_word(uint32_t c, uint32_t b, uint32_t lx, bool periodic) {
    const uint32_t mask = 0xffffffffu >> (32 - lx), sh = 32 - lx;
    if (!periodic) b &= 0x7fffffffu; /* bond bit 31 leads out of the word and is not used here */
    /* bonds j-1 -- j, then reversed so that leftward is upward */
    const uint32_t bl = periodic ? ((b << 1) | (b >> (lx - 1))) & mask : b << 1;
    const uint32_t up = carry_up(c, b, lx, periodic);
    const uint32_t dn = carry_up(__brev(c) >> sh, __brev(bl) >> sh, lx, periodic);
    return (up | (__brev(dn) >> sh)) & mask;
}

/* A block of words c[y + kGrowPitch z] (the odd pitch keeps both directions
 * free of bank conflicts) and its bonds: bx along x inside the word, by row y
 * to y + 1, bz plane z to z + 1; px / py / pz: the block spans the whole period
 * along x (one-word rows), y, z. */
constexpr uint32_t kGrowPitch = kGrowEdge + 1;
struct GrowBlock {
    uint32_t* c;
    const uint32_t *bx, *by, *bz;
    uint32_t lx; /* sites of a word */
    bool px, py, pz;
};

/* One axis of one word of a thread: position `lane` of line `line`.  up[k] / dn[k]
 * are the products of the bonds over the 2^k positions below / above, so a
 * scan along the line takes one shuffle and one operation per doubling step
 * and direction. */
struct GrowAxis {
    uint32_t up[5], dn[5];
    uint32_t at, below, above; /* the word, and those of the lines next to it */
    uint32_t lo, hi;           /* the bonds to them */
    uint32_t last;             /* the word after this axis' last scan */
    bool still;                /* that scan changed nothing in the line */

    /* si, sl: strides along the line and between lines; b bonds along it, bo across */
    __device__ __forceinline__ void start(uint32_t line, uint32_t si, uint32_t sl, const uint32_t* b, const uint32_t* bo,
                                          bool along, bool across) {
        constexpr uint32_t E = kGrowEdge;
        const uint32_t lane = threadIdx.x & 31u;
        at = lane * si + line * sl;
        below = line > 0 ? at - sl : at + (E - 1) * sl;
        above = line + 1 < E ? at + sl : at - (E - 1) * sl;
        up[0] = __shfl_sync(0xffffffffu, b[at], lane - 1);
        if (!along && lane == 0) up[0] = 0; /* products that would cross an open end are zero */
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            if (k < 4) up[k + 1] = up[k] & __shfl_sync(0xffffffffu, up[k], lane - (1u << k));
            dn[k] = __shfl_sync(0xffffffffu, up[k], lane + (1u << k));
        }
        lo = across || line > 0 ? bo[below] : 0u;
        hi = across || line + 1 < E ? bo[at] : 0u;
        last = 0;
        still = false;
    }

    /* One pass: the word takes the bits that reach it from the neighbouring
     * lines, its line is closed, and where it changed it is closed along x.
     * A line whose last scan changed nothing and which gets no new bits is
     * skipped.  Returns nonzero if the word changed. */
    __device__ __forceinline__ int pass(const GrowBlock& q) {
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t old = q.c[at];
        uint32_t v = old | (q.c[below] & lo) | (q.c[above] & hi);
        if (__all_sync(0xffffffffu, v == last) && still) return 0;
        uint32_t a = v, b = v;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            a |= up[k] & __shfl_sync(0xffffffffu, a, lane - (1u << k));
            b |= dn[k] & __shfl_sync(0xffffffffu, b, lane + (1u << k));
        }
        v = a | b;
        still = !__any_sync(0xffffffffu, v != old);
        if (!still) {
            v = close_word(v, q.bx[at], q.lx, q.px);
            if (v != old) q.c[at] = v;
        }
        last = v;
        return v != old;
    }
};

/* Closes the block (1024 / kT threads, kT lines of each axis per warp); c must
 * already be closed along x.  Passes alternate a scan of every line along y
 * with a scan of every line along z, each with one step along the other axis
 * and the closure along x; a pass that changes nothing ends it.  The bond
 * products stay in registers for all passes.  Returns the number of passes, or
 * 0 if max_pass passes were not enough (every pass that changes something sets
 * a bit, so 32^3 + 1 always are).  Bound by shuffles and shared loads (one warp
 * instruction per clock and SM): ten shuffles per line and pass. */
template <int kT>
__device__ __forceinline__ uint32_t close_block(const GrowBlock& q, uint32_t max_pass) {
    GrowAxis y[kT], z[kT];
#pragma unroll
    for (int p = 0; p < kT; ++p) {
        const uint32_t line = (threadIdx.x >> 5) + p * (kGrowEdge / kT);
        y[p].start(line, 1u, kGrowPitch, q.by, q.bz, q.py, q.pz);
        z[p].start(line, kGrowPitch, 1u, q.bz, q.by, q.pz, q.py);
    }
    for (uint32_t pass = 0; pass < max_pass; ++pass) {
        int changed = 0;
#pragma unroll
        for (int p = 0; p < kT; ++p) changed |= (pass & 1u) ? z[p].pass(q) : y[p].pass(q);
        if (!__syncthreads_or(changed)) return pass + 1;
    }
    return 0;
}

}  // namespace slsf

#endif /* SLSF_BITGROW_CUH */
