/*
 * Single-task kernels: the plain GPU path behind slsf_task_*.
 *
 *   k_init_random        ThetaModel::init (src/model.rs:373-377)
 *   k_metro_colour       one colour of metropolis_sweep_with_scratch
 *                        (src/updates.rs:440-486), one thread per Philox block
 *                        (two same-colour sites)
 *   k_metro_colour0_measure  colour 0 fused with the measurement of the state
 *                        it starts from (the batched grid path)
 *   k_wolff_tiles        per-site +x/+y/+z bond activation of
 *   k_wolff_boundary     wolff_cluster_step_with_theta_scratch
 *   k_wolff_flip         (src/updates.rs:551-620): components inside
 *                        32x8x4 tiles by union-find in shared memory, the
 *                        bonds between tiles by a lock-free global
 *                        union-find over the tile roots, then reflect the
 *                        seed's component
 *   k_measure            measure_theta_observables_with_scratch
 *                        (src/observables.rs:80-154), FP64 block sums, fixed
 *                        summation order (last block reduces the partials);
 *   k_measure_rows       the same with warps walking rows (L_x a multiple of
 *                        32): two sincos per site instead of four
 *
 * Metropolis and measurement here take the shapes that the patch walks of
 * kernel_walk.cu do not; the Wolff kernels lattices whose cluster is not grown
 * on bits (wolff_by_bits).
 * (The correlation functions are in kernel_corr.cu, batched over tasks.)
 */
#include <algorithm>

#include "engine.h"
#include "fastdiv.h"
#include "xy_device.cuh"

namespace slsf {

namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) k_init_random(float* __restrict__ theta, uint32_t volume,
                                                          uint64_t seed) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (4ull * q >= volume) return;
    const slsf_u32x4 b = slsf_stream(seed, 0, SLSF_PURPOSE_INIT, 0, q);
    const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t i = 4 * q + k;
        if (i < volume) theta[i] = slsf_angle_from_word(w[k]);
    }
}

/* Adds a per-thread count to stats[slot] with one global atomic per block
 * (warp sums, then a shared-memory sum): grid-wide kernels have tens of
 * thousands of warps, and one same-address atomic per warp serialises. */
__device__ __forceinline__ void block_count(uint32_t v, unsigned long long* stats, int slot) {
    __shared__ unsigned int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_sum, v);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(&stats[slot], (unsigned long long)s_sum);
}

/* Sums of the measurement (mx, my, J cos and J sin per axis) and where they
 * go: per-block partials, a block counter, the totals and an optional bin
 * row -- the last block adds the partials in block order. */
struct MeasureSink {
    double* partials;
    unsigned int* done;
    double* result;
    double* bin_row;
};

/* The last block's reduction of the per-block measurement partials into the
 * totals and the bin row (ThetaModel::measure's stream, src/model.rs:406-409,
 * in the batched kernels' column order). */
__device__ __forceinline__ void finish_measure(double (&acc)[8], double* scratch, const MeasureSink& m,
                                               uint32_t volume) {
    __shared__ bool last;
    block_sum<8>(acc, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) m.partials[blockIdx.x * 8 + k] = acc[k];
        __threadfence();
        last = (atomicAdd(m.done, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int k = 0; k < 8; ++k) tot[k] += ((volatile double*)m.partials)[b * 8 + k];
    block_sum<8>(tot, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) m.result[k] = tot[k];
        if (m.bin_row) {
            const double v = (double)volume;
            const double e = -(tot[2] + tot[3] + tot[4]) / v;
            const double vals[kBinCols] = {e,      e * e,  (tot[0] * tot[0] + tot[1] * tot[1]) / (v * v),
                                           tot[2], tot[3], tot[4],
                                           tot[5], tot[6], tot[7],
                                           tot[5] * tot[5], tot[6] * tot[6], tot[7] * tot[7]};
            for (int q = 0; q < kBinCols; ++q) m.bin_row[q] += vals[q];
        }
        *m.done = 0;
    }
}

/* Colour 0 of a sweep, grid-stride blocks, measuring the state it starts
 * from as the batched kernels do: every
 * bond has exactly one colour-0 end, so the three forward and three backward
 * bonds of the colour-0 sites and the magnetisation of each colour-0 site and
 * of its +x neighbour cover the lattice once; the FP32 bond terms are the
 * measurement kernels' (bond_cos / bond_sin), summed in FP64. */
template <bool kRecord>
__global__ void __launch_bounds__(kThreads)
    k_metro_colour(float* __restrict__ theta, const float* __restrict__ jxy,
                   const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz, float beta,
                   float width, uint64_t seed, uint64_t sweep, uint32_t colour, slsf_fastdiv div_hx,
                   slsf_fastdiv div_ly, unsigned long long* __restrict__ stats, uint8_t* __restrict__ record) {
    const uint32_t volume = lx * ly * lz;
    const uint32_t half = volume >> 1;
    const uint32_t npairs = (half + 1) >> 1;
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t accepted = 0;
    if (p < npairs) {
        const slsf_u32x4 blk = slsf_stream(seed, sweep, SLSF_PURPOSE_METRO, colour, p);
#pragma unroll
        for (uint32_t lane = 0; lane < 2; ++lane) {
            const uint32_t h = 2 * p + lane;
            if (h >= half) break;
            /* the h-th site of this colour: row = h / (L_x / 2) (x + L_x row = site index),
             * x = 2 (h mod L_x / 2) + (colour + y + z) mod 2; divisions as multiply-shifts */
            SiteXYZ s;
            const uint32_t row = slsf_fastdiv_div(h, div_hx), k = h - row * div_hx.d;
            s.z = slsf_fastdiv_div(row, div_ly);
            s.y = row - s.z * ly;
            s.x = 2u * k + ((colour + s.y + s.z) & 1u);
            s.idx = s.x + lx * row;
            uint32_t nb[6];
            neighbour_indices(s, lx, ly, lz, nb);
            float ns[6], nc[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) __sincosf(theta[nb[k]], &ns[k], &nc[k]);
            const float jx = jxy[s.z], jzp = jz[s.z], jzm = jz[s.z == 0 ? lz - 1 : s.z - 1];
            const float hx = field_component(jx, jzp, jzm, nc[0], nc[1], nc[2], nc[3], nc[4], nc[5]);
            const float hy = field_component(jx, jzp, jzm, ns[0], ns[1], ns[2], ns[3], ns[4], ns[5]);
            const float th = theta[s.idx];
            float si, ci;
            __sincosf(th, &si, &ci);
            float u_prop, u_acc;
            slsf_metro_uniforms(blk, lane, &u_prop, &u_acc);
            float tn, sn, cn;
            const bool acc = metro_decide(th, ci, si, hx, hy, beta, width, u_prop, u_acc, &tn, &sn, &cn);
            if (acc) {
                theta[s.idx] = tn;
                ++accepted;
            }
            if (kRecord) record[s.idx] = acc ? 1 : 0;
        }
    }
    block_count(accepted, stats, kStatAccepted);
}

__global__ void __launch_bounds__(kThreads, 3)
    k_metro_colour0_measure(float* __restrict__ theta, const float* __restrict__ jxy,
                   const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz, float beta,
                   float width, uint64_t seed, uint64_t sweep, uint32_t colour, slsf_fastdiv div_hx,
                   slsf_fastdiv div_ly, unsigned long long* __restrict__ stats, MeasureSink sink) {
    const uint32_t volume = lx * ly * lz;
    const uint32_t half = volume >> 1;
    const uint32_t npairs = (half + 1) >> 1;
    uint32_t accepted = 0;
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    auto pair = [&](uint32_t p) {
        const slsf_u32x4 blk = slsf_stream(seed, sweep, SLSF_PURPOSE_METRO, colour, p);
#pragma unroll
        for (uint32_t lane = 0; lane < 2; ++lane) {
            const uint32_t h = 2 * p + lane;
            if (h >= half) break;
            /* the h-th site of this colour: row = h / (L_x / 2) (x + L_x row = site index),
             * x = 2 (h mod L_x / 2) + (colour + y + z) mod 2; divisions as multiply-shifts */
            SiteXYZ s;
            const uint32_t row = slsf_fastdiv_div(h, div_hx), k = h - row * div_hx.d;
            s.z = slsf_fastdiv_div(row, div_ly);
            s.y = row - s.z * ly;
            s.x = 2u * k + ((colour + s.y + s.z) & 1u);
            s.idx = s.x + lx * row;
            uint32_t nb[6];
            neighbour_indices(s, lx, ly, lz, nb);
            float ns[6], nc[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) __sincosf(theta[nb[k]], &ns[k], &nc[k]);
            const float jx = jxy[s.z], jzp = jz[s.z], jzm = jz[s.z == 0 ? lz - 1 : s.z - 1];
            const float hx = field_component(jx, jzp, jzm, nc[0], nc[1], nc[2], nc[3], nc[4], nc[5]);
            const float hy = field_component(jx, jzp, jzm, ns[0], ns[1], ns[2], ns[3], ns[4], ns[5]);
            const float th = theta[s.idx];
            float si, ci;
            __sincosf(th, &si, &ci);
            {
                /* neighbours in the order +x -x +y -y +z -z; a backward bond
                 * starts at the neighbour (its layer's coupling for z) */
                acc[0] += (double)ci + (double)nc[0];
                acc[1] += (double)si + (double)ns[0];
                acc[2] += (double)bond_cos(jx, ci, si, nc[0], ns[0]) + (double)bond_cos(jx, nc[1], ns[1], ci, si);
                acc[3] += (double)bond_cos(jx, ci, si, nc[2], ns[2]) + (double)bond_cos(jx, nc[3], ns[3], ci, si);
                acc[4] += (double)bond_cos(jzp, ci, si, nc[4], ns[4]) + (double)bond_cos(jzm, nc[5], ns[5], ci, si);
                acc[5] += (double)bond_sin(jx, ci, si, nc[0], ns[0]) + (double)bond_sin(jx, nc[1], ns[1], ci, si);
                acc[6] += (double)bond_sin(jx, ci, si, nc[2], ns[2]) + (double)bond_sin(jx, nc[3], ns[3], ci, si);
                acc[7] += (double)bond_sin(jzp, ci, si, nc[4], ns[4]) + (double)bond_sin(jzm, nc[5], ns[5], ci, si);
            }
            float u_prop, u_acc;
            slsf_metro_uniforms(blk, lane, &u_prop, &u_acc);
            float tn, sn, cn;
            const bool ok = metro_decide(th, ci, si, hx, hy, beta, width, u_prop, u_acc, &tn, &sn, &cn);
            if (ok) {
                theta[s.idx] = tn;
                ++accepted;
            }
        }
    };
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npairs; p += gridDim.x * blockDim.x) pair(p);
    block_count(accepted, stats, kStatAccepted);
    __shared__ double scratch[8 * 32];
    finish_measure(acc, scratch, sink, volume);
}

/* Wolff tiles: a CTA labels one tile of kTileX x kTileY x kTileZ sites. */
constexpr uint32_t kTileX = 32, kTileY = 8, kTileZ = 4;
constexpr uint32_t kTileSites = kTileX * kTileY * kTileZ;
static_assert(kTileX == 32, "a tile row is one warp");

inline uint32_t wolff_tiles(const TaskView& t) {
    return ((t.lx + kTileX - 1) / kTileX) * ((t.ly + kTileY - 1) / kTileY) * ((t.lz + kTileZ - 1) / kTileZ);
}

/* Lattices whose Wolff update grows the seed's cluster on bit-packed bonds
 * (kernel_wolff_bits.cu) instead of labelling 32x8x4 tiles: from 2^21 sites,
 * where that is the shorter of the two.  The tiles take 30 ns each, whatever
 * the lattice's form.  The growth is a chain of region closures, half the
 * regions of each axis one after the other, 11 us each (5.5 us for every region
 * of L_x / 32 + L_y / 32 + L_z / 32), and 6 us per 2^20 sites for the bonds and
 * the reflection.  Measured on B200, us per Wolff update at T = 1.2, bits against
 * tiles: 128^3 110 / 106, 150x150x100 116 / 125, 160^3 131 / 169, 256^3 257 / 562,
 * 128x128x1024 309 / 613, 1024x1024x16 440 / 546; 2048x32x32 346 / 106,
 * 1024x1024x2 256 / 117, 512x512x8 182 / 104, 32x32x4096 483 / 179, 64x64x1024
 * 227 / 185. */
constexpr uint64_t kWolffBitsMinSites = 1u << 21;
constexpr uint64_t kRegionTiles = 180, kTileSitesByBits = 5400; /* tiles' worth of a region; sites by bits in a tile's time */

inline bool wolff_by_bits(const TaskView& t) {
    const uint64_t v = (uint64_t)t.lx * t.ly * t.lz;
    const uint64_t chain = (uint64_t)(t.lx + 31) / 32 + (t.ly + 31) / 32 + (t.lz + 31) / 32;
    return v >= kWolffBitsMinSites && kRegionTiles * chain + v / kTileSitesByBits < wolff_tiles(t) &&
           wolff_bits_scratch_bytes(t.lx, t.ly, t.lz) <= 4ull * v;
}

/* ---- Wolff: union-find with links down a total order of the nodes ---- */

/* Loop bounds of the union-find: parents are at most their children in the
 * order, so a path has at most `volume` steps and a union, which takes one down one of two
 * paths each time round, at most twice as many.  A nonzero `limit`
 * (slsf_ctx_set_loop_limit) lowers both, to exercise the error path. */
struct UfBounds {
    uint32_t find;
    uint64_t uni;
};

__device__ __forceinline__ UfBounds uf_bounds(uint32_t volume, uint32_t limit) {
    const uint64_t u = 2ull * volume + 2;
    return {limit ? min(limit, volume) : volume, limit && limit < u ? limit : u};
}

/* Lock-free union after Rem (Dijkstra, A Discipline of Programming, 1976; with
 * splicing, Patwary, Blair and Manne 2010): climb both paths together, always
 * from the node with the larger parent; a root is hooked under the other's
 * parent by a CAS, any other node is pointed there as it is left (both belong
 * to one component once this union is done, and parents stay below their
 * children, so a store that another overtakes loses nothing but a shortcut).
 * One dependent read a step, where finding both roots first took four: those
 * reads of the global array, 300 ns each, are the time of k_wolff_boundary.
 *
 * The order is that of the indices in a tile (kScatter false), where a warp's
 * runs are short, and that of a bijective hash of them between the tiles: a
 * row of tiles ordered by index hangs every root on its neighbour's, a chain
 * as long as the row that the union across the period and every thread of the
 * reflection climb, while a random order (Goel, Khanna, Larkin and Tarjan,
 * Disjoint set union with randomized linking, 2014) keeps the expected depth
 * logarithmic. */
template <bool kScatter>
__device__ __forceinline__ uint32_t uf_order(uint32_t i) {
    return kScatter ? i * 2654435769u : i; /* odd factor, 2^32 / golden ratio */
}

template <bool kScatter>
__device__ __forceinline__ bool uf_union(uint32_t* parent, uint32_t a, uint32_t b, uint64_t bound) {
    volatile uint32_t* par = parent;
    uint32_t pa = par[a], pb = par[b];
    for (uint64_t it = 0; it < bound; ++it) {
        if (pa == pb) return true;
        if (uf_order<kScatter>(pa) < uf_order<kScatter>(pb)) {
            const uint32_t t = a, pt = pa;
            a = b, pa = pb;
            b = t, pb = pt;
        }
        if (pa == a) { /* a root, as last read */
            pa = atomicCAS(&parent[a], a, pb);
            if (pa == a) return true;
        } else {
            par[a] = pb;
            a = pa;
            pa = par[a];
        }
    }
    return false;
}

/* Two rows a warp and phase: the unions' chains run side by side (us per call of
 * Metropolis and Wolff on 256 / 512 / 1024 threads: 48^3 83 / 76 / 74, 100x12x138
 * 87 / 81 / 79, 128^3 - / 141 / 152). */
constexpr int kTileThreads = 512;

/* Root of x in a tile's shared array, splitting the path. */
__device__ __forceinline__ uint32_t tile_find(uint32_t* lpar, uint32_t x, uint32_t bound, bool* ok) {
    volatile uint32_t* par = lpar;
    uint32_t p = par[x];
    for (uint32_t it = 0; it <= bound; ++it) {
        if (p == x) return x;
        const uint32_t gp = par[p];
        if (gp == p) return p;
        par[x] = gp;
        x = p;
        p = gp;
    }
    *ok = false;
    return x;
}

/* Bond activation (try_add_wolff_neighbor, src/updates.rs:537-548) for every
 * site of a tile, then the tile's components over its inner bonds: each site
 * gets parent = the smallest site of its component inside the tile (local
 * order is global order inside a tile, so parent[i] <= i holds).  Bonds that
 * leave the tile are joined by k_wolff_boundary. */
__global__ void __launch_bounds__(kTileThreads)
    k_wolff_tiles(const float* __restrict__ theta, const float* __restrict__ jxy,
                  const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz,
                  float minus_two_beta, float phi, uint64_t seed, uint64_t counter,
                  uint8_t* __restrict__ bonds, uint32_t* __restrict__ parent,
                  unsigned long long* __restrict__ stats, uint32_t limit) {
    __shared__ uint32_t lpar[kTileSites];
    const UfBounds bd = uf_bounds(kTileSites, limit);
    __shared__ uint8_t lbits[kTileSites];
    const uint32_t ntx = (lx + kTileX - 1) / kTileX, nty = (ly + kTileY - 1) / kTileY;
    const uint32_t tx = blockIdx.x % ntx, rest = blockIdx.x / ntx;
    const uint32_t ty = rest % nty, tz = rest / nty;
    const uint32_t x0 = tx * kTileX, y0 = ty * kTileY, z0 = tz * kTileZ;
    const uint32_t ex = min(kTileX, lx - x0), ey = min(kTileY, ly - y0), ez = min(kTileZ, lz - z0);
    const uint32_t plane = lx * ly, volume = plane * lz;
    float sphi, cphi;
    __sincosf(phi, &sphi, &cphi);
    auto proj = [&](uint32_t site) {
        float sn, cn;
        __sincosf(theta[site], &sn, &cn);
        return wolff_projection(cn, sn, cphi, sphi);
    };
    for (uint32_t l = threadIdx.x; l < kTileSites; l += blockDim.x) {
        const uint32_t ax = l % kTileX, ay = (l / kTileX) % kTileY, az = l / (kTileX * kTileY);
        uint32_t bits = 0;
        if (ax < ex && ay < ey && az < ez) {
            const uint32_t x = x0 + ax, y = y0 + ay, z = z0 + az;
            const uint32_t i = x + lx * (y + ly * z);
            const uint32_t xp = (x + 1 == lx) ? i + 1 - lx : i + 1;
            const uint32_t yp = (y + 1 == ly) ? i + lx - plane : i + lx;
            const uint32_t zp = (z + 1 == lz) ? i + plane - volume : i + plane;
            const float ri = proj(i);
            const slsf_u32x4 b = slsf_stream(seed, counter, SLSF_PURPOSE_WOLFF_BOND, 0, i);
            if (wolff_bond_active(jxy[z], ri, proj(xp), minus_two_beta, b.x)) bits |= 1u;
            if (wolff_bond_active(jxy[z], ri, proj(yp), minus_two_beta, b.y)) bits |= 2u;
            if (wolff_bond_active(jz[z], ri, proj(zp), minus_two_beta, b.z)) bits |= 4u;
            bonds[i] = (uint8_t)bits;
        }
        lbits[l] = (uint8_t)bits;
        /* A warp holds one row of the tile (kTileX == 32 sites, lane = x):
         * the sites joined along x form runs, and every site's parent is the
         * first site of its run (the highest run start at or below its lane),
         * so the x bonds inside the tile need no union. */
        const unsigned xb = __ballot_sync(0xffffffffu, (bits & 1u) && ax + 1 < ex);
        const unsigned starts = ~(xb << 1);
        const uint32_t lane = l % kTileX;
        const unsigned upto = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
        lpar[l] = l - lane + (31u - __clz(starts & upto));
    }
    __syncthreads();
    bool ok = true;
    for (uint32_t l = threadIdx.x; l < kTileSites; l += blockDim.x) {
        /* a warp holds one row (lane = x); a y or z bond whose left neighbour's
         * bond joins the same two x-runs adds nothing, so only the first bond of
         * each such stretch unions */
        const uint32_t lane = l % kTileX, bits = lbits[l];
        const uint32_t ay = (l / kTileX) % kTileY, az = l / (kTileX * kTileY);
        const bool yin = ay + 1 < ey, zin = az + 1 < ez; /* warp-uniform */
        const bool xin = lane + 1 < ex;
        const unsigned own = __ballot_sync(0xffffffffu, (bits & 1u) && xin);
        const unsigned yb = __ballot_sync(0xffffffffu, (bits & 2u) && yin);
        const unsigned zb = __ballot_sync(0xffffffffu, (bits & 4u) && zin);
        const unsigned yrow = yin ? __ballot_sync(0xffffffffu, (lbits[l + kTileX] & 1u) && xin) : 0u;
        const unsigned zrow = zin ? __ballot_sync(0xffffffffu, (lbits[l + kTileX * kTileY] & 1u) && xin) : 0u;
        const unsigned ylead = yb & ~((yb & own & yrow) << 1), zlead = zb & ~((zb & own & zrow) << 1);
        if ((ylead >> lane) & 1u) ok &= uf_union<false>(lpar, l, l + kTileX, bd.uni);
        if ((zlead >> lane) & 1u) ok &= uf_union<false>(lpar, l, l + kTileX * kTileY, bd.uni);
    }
    __syncthreads();
    for (uint32_t l = threadIdx.x; l < kTileSites; l += blockDim.x) {
        const uint32_t ax = l % kTileX, ay = (l / kTileX) % kTileY, az = l / (kTileX * kTileY);
        if (ax >= ex || ay >= ey || az >= ez) continue;
        const uint32_t r = tile_find(lpar, l, bd.find, &ok);
        const uint32_t rx = r % kTileX, ry = (r / kTileX) % kTileY, rz = r / (kTileX * kTileY);
        const uint32_t i = (x0 + ax) + lx * ((y0 + ay) + ly * (z0 + az));
        parent[i] = (x0 + rx) + lx * ((y0 + ry) + ly * (z0 + rz));
    }
    if (!ok) atomicOr(&stats[kStatError], kErrUnionFindLimit);
}

/* The active bonds that leave a tile (its last x, y or z; periodic wraps
 * included), joined in the global union-find over the tile roots.  A warp
 * takes one face row of one tile: the 8 x 4 bonds of the +x face (lane =
 * y + 8 z), one of the 4 rows of the +y face or one of the 8 rows of the +z
 * face (lane = x).  The bonds of a face row mostly join the same few pairs of
 * tile roots, so the lanes group them by (root, root) pair and one lane per
 * pair joins. */
constexpr uint32_t kFaceRows = 1 + kTileZ + kTileY;
static_assert(kTileY * kTileZ == 32, "an x face is one warp");

__global__ void __launch_bounds__(kThreads)
    k_wolff_boundary(const uint8_t* __restrict__ bonds, uint32_t lx, uint32_t ly, uint32_t lz, uint32_t n_tiles,
                     uint32_t* parent, unsigned long long* stats, uint32_t limit) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t tile = w / kFaceRows, item = w - tile * kFaceRows;
    if (tile >= n_tiles) return; /* whole warps */
    const uint32_t ntx = (lx + kTileX - 1) / kTileX, nty = (ly + kTileY - 1) / kTileY;
    const uint32_t tx = tile % ntx, rest = tile / ntx, ty = rest % nty, tz = rest / nty;
    const uint32_t x0 = tx * kTileX, y0 = ty * kTileY, z0 = tz * kTileZ;
    const uint32_t ex = min(kTileX, lx - x0), ey = min(kTileY, ly - y0), ez = min(kTileZ, lz - z0);
    const uint32_t plane = lx * ly, volume = plane * lz;
    uint32_t ax, ay, az, d;
    if (item == 0) {
        d = 0, ax = ex - 1, ay = lane % kTileY, az = lane / kTileY;
    } else if (item <= kTileZ) {
        d = 1, ax = lane, ay = ey - 1, az = item - 1;
    } else {
        d = 2, ax = lane, ay = item - 1 - kTileZ, az = ez - 1;
    }
    const bool in = ax < ex && ay < ey && az < ez;
    const uint32_t x = x0 + ax, y = y0 + ay, z = z0 + az;
    const uint32_t i = in ? x + lx * (y + ly * z) : 0u;
    const bool act = in && (bonds[i] & (1u << d));
    uint32_t a = 0, b = 0;
    if (act) {
        const uint32_t nb = d == 0   ? ((x + 1 == lx) ? i + 1 - lx : i + 1)
                            : d == 1 ? ((y + 1 == ly) ? i + lx - plane : i + lx)
                                     : ((z + 1 == lz) ? i + plane - volume : i + plane);
        a = parent[i];
        b = parent[nb];
    }
    const unsigned long long key = act ? (((unsigned long long)a << 32) | b) : ~0ull;
    const unsigned grp = __match_any_sync(0xffffffffu, key);
    bool ok = true;
    if (act && lane == (uint32_t)(__ffs(grp) - 1) && a != b) ok = uf_union<true>(parent, a, b, uf_bounds(volume, limit).uni);
    if (!ok) atomicOr(&stats[kStatError], kErrUnionFindLimit);
}

/* Reflect the seed's component (src/updates.rs:602-617).  A site's parent is
 * its tile's root, which reaches the component's root in the few steps that
 * the joins left; the array no longer changes, so every chain ends there.
 * Finding the roots here, where the tiles' few roots come from the cache,
 * saves a kernel that shortened the chains first (4.8 us of 58 at 64^3). */
__global__ void __launch_bounds__(kThreads)
    k_wolff_flip(float* __restrict__ theta, uint32_t volume, const uint32_t* __restrict__ parent, uint32_t seed_idx,
                 float phi, unsigned long long* stats, uint8_t* __restrict__ cluster_out, uint32_t limit) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t bound = uf_bounds(volume, limit).find;
    bool ok = true;
    auto root_of = [&](uint32_t x) {
        for (uint32_t it = 0; it <= bound; ++it) {
            const uint32_t p = parent[x];
            if (p == x) return x;
            x = p;
        }
        ok = false;
        return x;
    };
    uint32_t in = 0;
    if (i < volume) {
        in = root_of(i) == root_of(seed_idx) ? 1u : 0u;
        if (!ok) atomicOr(&stats[kStatError], kErrUnionFindLimit);
        if (in) theta[i] = slsf_reflect(theta[i], phi);
        if (cluster_out) cluster_out[i] = (uint8_t)in;
    }
    block_count(in, stats, kStatClusterSites);
}

/* ---- fused observables ---- */
constexpr int kMeasureThreads = 256;

__global__ void __launch_bounds__(kMeasureThreads)
    k_measure(const float* __restrict__ theta, const float* __restrict__ jxy,
              const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz, slsf_fastdiv div_lx,
              slsf_fastdiv div_ly, double* __restrict__ partials, unsigned int* __restrict__ done,
              double* __restrict__ result, double* __restrict__ bin_row) {
    __shared__ double scratch[8 * 32];
    __shared__ bool last;
    const uint32_t volume = lx * ly * lz, plane = lx * ly;
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < volume; i += stride) {
        const uint32_t row = slsf_fastdiv_div(i, div_lx), z = slsf_fastdiv_div(row, div_ly);
        const uint32_t x = i - row * lx, y = row - z * ly;
        const uint32_t ix = (x + 1 == lx) ? i + 1 - lx : i + 1;
        const uint32_t iy = (y + 1 == ly) ? i + lx - plane : i + lx;
        const uint32_t iz = (z + 1 == lz) ? i + plane - volume : i + plane;
        float si, ci, sx, cx, sy, cy, sz, cz;
        __sincosf(theta[i], &si, &ci);
        __sincosf(theta[ix], &sx, &cx);
        __sincosf(theta[iy], &sy, &cy);
        __sincosf(theta[iz], &sz, &cz);
        const float jx = jxy[z], jzz = jz[z];
        /* diff_cos_sin (src/observables.rs:9-11): cos(a-b), sin(a-b) from trig. */
        acc[0] += ci;
        acc[1] += si;
        acc[2] += bond_cos(jx, ci, si, cx, sx);
        acc[3] += bond_cos(jx, ci, si, cy, sy);
        acc[4] += bond_cos(jzz, ci, si, cz, sz);
        acc[5] += bond_sin(jx, ci, si, cx, sx);
        acc[6] += bond_sin(jx, ci, si, cy, sy);
        acc[7] += bond_sin(jzz, ci, si, cz, sz);
    }
    block_sum<8>(acc, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) partials[blockIdx.x * 8 + k] = acc[k];
        __threadfence();
        last = (atomicAdd(done, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    /* Last block: sum the per-block partials in block order. */
    __threadfence();
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int k = 0; k < 8; ++k) tot[k] += ((volatile double*)partials)[b * 8 + k];
    block_sum<8>(tot, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) result[k] = tot[k];
        if (bin_row) {
            /* ThetaModel::measure's stream (src/model.rs:406-409) added to
             * the bin's sums, in the batched kernels' column order. */
            const double v = (double)volume;
            const double e = -(tot[2] + tot[3] + tot[4]) / v;
            const double vals[kBinCols] = {e,      e * e,  (tot[0] * tot[0] + tot[1] * tot[1]) / (v * v),
                                           tot[2], tot[3], tot[4],
                                           tot[5], tot[6], tot[7],
                                           tot[5] * tot[5], tot[6] * tot[6], tot[7] * tot[7]};
            for (int q = 0; q < kBinCols; ++q) bin_row[q] += vals[q];
        }
        *done = 0;
    }
}

/* The same measurement for L_x a multiple of 32 and L_y a multiple of 16:
 * a warp owns word k (lane = x - 32 k) of plane z for a run of 16 rows and
 * walks it along y, so each site's own trig is the previous row's +y trig:
 * two sincos per site (+y, +z) instead of four, the +x neighbour by shuffle.
 * Identical FP32 bond terms; FP64 sums in another order. */
constexpr uint32_t kMeasureSeg = 16;

__global__ void __launch_bounds__(kMeasureThreads)
    k_measure_rows(const float* __restrict__ theta, const float* __restrict__ jxy,
                   const float* __restrict__ jz, uint32_t lx, uint32_t ly, uint32_t lz,
                   double* __restrict__ partials, unsigned int* __restrict__ done,
                   double* __restrict__ result, double* __restrict__ bin_row) {
    __shared__ double scratch[8 * 32];
    __shared__ bool last;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t words = lx >> 5, nseg = ly / kMeasureSeg, plane = lx * ly, volume = plane * lz;
    const uint32_t units = words * nseg * lz;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
        const uint32_t k = u % words, rest = u / words, sg = rest % nseg, z = rest / nseg;
        const uint32_t x = 32u * k + lane, xn = (k + 1 == words) ? 0u : 32u * (k + 1);
        const uint32_t zbase = z * plane, zp_base = (z + 1 == lz) ? 0u : (z + 1) * plane;
        const float jx = jxy[z], jzz = jz[z];
        const uint32_t y0 = sg * kMeasureSeg;
        float si, ci;
        __sincosf(theta[zbase + y0 * lx + x], &si, &ci);
        /* the angles of the next row's loads, one row ahead */
        auto yrow = [&](uint32_t y) { return (y + 1 == ly) ? 0u : y + 1; };
        float t_yp = theta[zbase + yrow(y0) * lx + x], t_zp = theta[zp_base + y0 * lx + x];
        float t_xn = theta[zbase + y0 * lx + xn];
        for (uint32_t y = y0; y < y0 + kMeasureSeg; ++y) {
            const uint32_t row = zbase + y * lx;
            const float a_yp = t_yp, a_zp = t_zp, a_xn = t_xn;
            if (y + 1 < y0 + kMeasureSeg) {
                t_yp = theta[zbase + yrow(y + 1) * lx + x];
                t_zp = theta[zp_base + (y + 1) * lx + x];
                t_xn = theta[row + lx + xn];
            }
            float sx, cx, sy, cy, sz, cz, sn, cn;
            __sincosf(a_yp, &sy, &cy);
            __sincosf(a_zp, &sz, &cz);
            __sincosf(a_xn, &sn, &cn);
            sx = __shfl_sync(0xffffffffu, si, (lane + 1u) & 31u);
            cx = __shfl_sync(0xffffffffu, ci, (lane + 1u) & 31u);
            if (lane == 31) {
                sx = sn;
                cx = cn;
            }
            acc[0] += ci;
            acc[1] += si;
            acc[2] += bond_cos(jx, ci, si, cx, sx);
            acc[3] += bond_cos(jx, ci, si, cy, sy);
            acc[4] += bond_cos(jzz, ci, si, cz, sz);
            acc[5] += bond_sin(jx, ci, si, cx, sx);
            acc[6] += bond_sin(jx, ci, si, cy, sy);
            acc[7] += bond_sin(jzz, ci, si, cz, sz);
            si = sy;
            ci = cy;
        }
    }
    block_sum<8>(acc, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) partials[blockIdx.x * 8 + k] = acc[k];
        __threadfence();
        last = (atomicAdd(done, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int k = 0; k < 8; ++k) tot[k] += ((volatile double*)partials)[b * 8 + k];
    block_sum<8>(tot, scratch);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 8; ++k) result[k] = tot[k];
        if (bin_row) {
            const double v = (double)volume;
            const double e = -(tot[2] + tot[3] + tot[4]) / v;
            const double vals[kBinCols] = {e,      e * e,  (tot[0] * tot[0] + tot[1] * tot[1]) / (v * v),
                                           tot[2], tot[3], tot[4],
                                           tot[5], tot[6], tot[7],
                                           tot[5] * tot[5], tot[6] * tot[6], tot[7] * tot[7]};
            for (int q = 0; q < kBinCols; ++q) bin_row[q] += vals[q];
        }
        *done = 0;
    }
}

inline bool measure_rows_supported(uint32_t lx, uint32_t ly) { return lx % 32 == 0 && ly % kMeasureSeg == 0; }

inline uint32_t blocks_for(uint64_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

}  // namespace

namespace {

/* One block per source array; coalesced copy into the contiguous output. */
__global__ void k_gather(const double* const* __restrict__ src, uint32_t per, double* __restrict__ dst) {
    const double* s = src[blockIdx.x];
    double* d = dst + (size_t)blockIdx.x * per;
    for (uint32_t k = threadIdx.x; k < per; k += blockDim.x) d[k] = s[k];
}

struct Couplings {
    float xy[kCouplingsPerLaunch], z[kCouplingsPerLaunch];
};

__global__ void k_set_couplings(float* __restrict__ jxy, float* __restrict__ jz, uint32_t n, const __grid_constant__ Couplings c) {
    if (threadIdx.x >= n) return;
    jxy[threadIdx.x] = c.xy[threadIdx.x];
    jz[threadIdx.x] = c.z[threadIdx.x];
}

__global__ void k_publish_stats(unsigned long long* __restrict__ stats, unsigned long long* __restrict__ host) {
    const unsigned long long v = stats[threadIdx.x];
    host[threadIdx.x] = v;
    stats[threadIdx.x] = 0;
}

}  // namespace

uint32_t set_couplings_launches(uint32_t lz) {
    const uint32_t n = (lz + kCouplingsPerLaunch - 1) / kCouplingsPerLaunch;
    return n <= kCouplingsLaunches ? n : 0;
}

cudaError_t launch_set_couplings(float* jxy, float* jz, const float* j, uint32_t lz, cudaStream_t s) {
    if (set_couplings_launches(lz) == 0) {
        const cudaError_t e = cudaMemcpyAsync(jxy, j, 4ull * lz, cudaMemcpyHostToDevice, s);
        return e != cudaSuccess ? e : cudaMemcpyAsync(jz, j + lz, 4ull * lz, cudaMemcpyHostToDevice, s);
    }
    for (uint32_t lo = 0; lo < lz; lo += kCouplingsPerLaunch) {
        const uint32_t n = std::min(kCouplingsPerLaunch, lz - lo);
        Couplings c = {};
        std::copy(j + lo, j + lo + n, c.xy);
        std::copy(j + lz + lo, j + lz + lo + n, c.z);
        k_set_couplings<<<1, kCouplingsPerLaunch, 0, s>>>(jxy + lo, jz + lo, n, c);
    }
    return cudaGetLastError();
}

void launch_publish_stats(unsigned long long* stats, unsigned long long* host, cudaStream_t s) {
    k_publish_stats<<<1, kStatSlots, 0, s>>>(stats, host);
}

void launch_gather(const double* const* src, uint32_t n, uint32_t per, double* dst, cudaStream_t s) {
    k_gather<<<n, 128, 0, s>>>(src, per, dst);
}

void launch_init_random(float* theta, uint32_t volume, uint64_t seed, cudaStream_t s) {
    const uint32_t quads = (volume + 3) / 4;
    k_init_random<<<blocks_for(quads, kThreads), kThreads, 0, s>>>(theta, volume, seed);
}

void launch_metro_colour(const TaskView& t, uint64_t sweep, uint32_t colour, uint8_t* record,
                         cudaStream_t s) {
    if (!record && walk_supports(t)) {
        launch_walk_colour(t, sweep, colour, false, nullptr, s);
        return;
    }
    const uint32_t volume = t.lx * t.ly * t.lz;
    const uint32_t npairs = ((volume >> 1) + 1) >> 1;
    const uint32_t grid = blocks_for(npairs, kThreads);
    const slsf_fastdiv dhx = slsf_fastdiv_make(t.lx / 2), dly = slsf_fastdiv_make(t.ly);
    if (record)
        k_metro_colour<true><<<grid, kThreads, 0, s>>>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, t.beta, t.width,
                                                       t.seed, sweep, colour, dhx, dly, t.stats, record);
    else
        k_metro_colour<false><<<grid, kThreads, 0, s>>>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, t.beta, t.width,
                                                        t.seed, sweep, colour, dhx, dly, t.stats, nullptr);
}

void launch_metro_colour0_measure(const TaskView& t, uint64_t sweep, double* bin_row, cudaStream_t s) {
    if (walk_supports(t)) {
        launch_walk_colour(t, sweep, 0, true, bin_row, s);
        return;
    }
    const uint32_t volume = t.lx * t.ly * t.lz;
    const uint32_t npairs = ((volume >> 1) + 1) >> 1;
    /* grid-stride blocks, as many as stay resident (at most kMeasureMaxBlocks,
     * the partials' rows); a fixed count per device keeps the sums' order */
    static int per_sm = 0;
    if (per_sm == 0 &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_metro_colour0_measure, kThreads, 0) !=
            cudaSuccess)
        per_sm = 1;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t cap = (uint32_t)std::max(1, std::min(per_sm * sms, kMeasureMaxBlocks));
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(blocks_for(npairs, kThreads), cap));
    const slsf_fastdiv dhx = slsf_fastdiv_make(t.lx / 2), dly = slsf_fastdiv_make(t.ly);
    const MeasureSink sink = {t.partials, t.done, t.result, bin_row};
    k_metro_colour0_measure<<<grid, kThreads, 0, s>>>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, t.beta, t.width,
                                                      t.seed, sweep, 0, dhx, dly, t.stats, sink);
}

int launch_wolff(const TaskView& t, uint64_t counter, uint8_t* bonds, uint32_t* parent,
                 uint8_t* cluster_out, cudaStream_t s, float* phi_out, uint32_t seed_site[3], bool record_bonds) {
    /* the bit planes live in the union-find array */
    if (wolff_by_bits(t))
        return launch_wolff_bits(t, counter, parent, record_bonds ? bonds : nullptr, cluster_out, s, phi_out,
                                 seed_site);
    /* The reflection axis and seed site (src/updates.rs:564-568) come from
     * the WOLFF_PICK block, computed here on the host from the same header. */
    const slsf_u32x4 pick = slsf_stream(t.seed, counter, SLSF_PURPOSE_WOLFF_PICK, 0, 0);
    const float phi = slsf_angle_from_word(pick.x);
    const uint32_t x0 = slsf_range(pick.y, t.lx), y0 = slsf_range(pick.z, t.ly), z0 = slsf_range(pick.w, t.lz);
    const uint32_t volume = t.lx * t.ly * t.lz;
    const uint32_t seed_idx = x0 + t.lx * (y0 + t.ly * z0);
    const uint32_t grid = blocks_for(volume, kThreads);
    const uint32_t tiles = wolff_tiles(t);
    k_wolff_tiles<<<tiles, kTileThreads, 0, s>>>(t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, -2.0f * t.beta, phi,
                                             t.seed, counter, bonds, parent, t.stats, t.loop_limit);
    k_wolff_boundary<<<blocks_for((uint64_t)tiles * kFaceRows * 32, kThreads), kThreads, 0, s>>>(
        bonds, t.lx, t.ly, t.lz, tiles, parent, t.stats, t.loop_limit);
    k_wolff_flip<<<grid, kThreads, 0, s>>>(t.theta, volume, parent, seed_idx, phi, t.stats, cluster_out, t.loop_limit);
    if (phi_out) *phi_out = phi;
    if (seed_site) {
        seed_site[0] = x0;
        seed_site[1] = y0;
        seed_site[2] = z0;
    }
    return 3;
}

int measure_partial_blocks(uint32_t volume) {
    return (int)std::max<uint32_t>(1, std::min<uint32_t>(blocks_for(volume, kMeasureThreads), kMeasureMaxBlocks));
}

void launch_measure(const TaskView& t, double* bin_row, cudaStream_t s) {
    if (walk_supports(t)) {
        launch_walk_measure(t, bin_row, s);
        return;
    }
    const uint32_t volume = t.lx * t.ly * t.lz;
    if (measure_rows_supported(t.lx, t.ly)) {
        k_measure_rows<<<measure_partial_blocks(volume), kMeasureThreads, 0, s>>>(
            t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, t.partials, t.done, t.result, bin_row);
        return;
    }
    k_measure<<<measure_partial_blocks(volume), kMeasureThreads, 0, s>>>(
        t.theta, t.jxy, t.jz, t.lx, t.ly, t.lz, slsf_fastdiv_make(t.lx), slsf_fastdiv_make(t.ly), t.partials, t.done,
        t.result, bin_row);
}

}  // namespace slsf
