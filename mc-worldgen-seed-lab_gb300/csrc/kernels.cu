/* kernels.cu -- sm_103a kernels of the biome path and their host launchers.
 *
 *  per-seed setup   k_setup_xo      one thread per (seed, lattice): Xoroshiro positional seeding and the
 *                                   256-step Fisher-Yates shuffle in a bank-conflict-free shared layout
 *                   k_setup_legacy  Nether biome noises: java.util.Random, octaves from the zero octave down
 *                   k_setup_end     End island simplex: LCG(seed) jumped 17292 steps, one shuffle
 *  per-point        k_points        seeds x quart points (ENGINE tie rule), lattices read through L1
 *                   k_grid          the Nether's quart grid, lattices staged in shared memory;
 *                                   ENGINE biomes or GRID_CHAIN records (leaf, fitness, tie flag, target)
 *                   (the Overworld's grids and block maps: owtile.cu)
 *                   k_chain_resolve GRID_CHAIN replay for the (rare) tied cells
 *                   k_blockgrid     libmcgen mcgen_biome_grid: BiomeManager zoom + chunk-cell tie chain
 *                   k_end_chunks    End island class per chunk, tiles of chunks (endtile.cuh)
 *                   k_end_samples, k_block_points  sparse End samples, block points: one per warp
 */
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include "climate.cuh"
#include "endtile.cuh"
#include "device.cuh"
#include "launch.h"
#include "legacy.cuh"
#include "batch.h"
#include "prof.h"
#include "warpcell.cuh"

using namespace mgd;

/* the cooperative 16-byte copies below rely on these layouts */
static_assert(sizeof(MgLattice) % 16 == 0, "lattice size");
static_assert(sizeof(MgSpline) % 16 == 0, "spline size");
static_assert(offsetof(MgWorldDesc, spline) % 16 == 0, "spline alignment in the description");
static_assert(sizeof(MgWorldDesc) <= 24576, "world description must fit the kernel parameter space");

namespace mg {

static long long g_launches = 0;
long long launch_count() { return g_launches; }
static inline void count_launch() { __atomic_add_fetch(&g_launches, 1, __ATOMIC_RELAXED); }
void count_launch_external() { count_launch(); }

/* ============================================================================ per-seed setup */
#define SETUP_NT 128
/* Shuffle state of thread t: byte i lives in byte (i & 3) of word perm[i >> 2][t], so every access of a
 * thread hits bank t % 32 whatever i is: the 32 lanes of a warp never conflict. */
__device__ __forceinline__ void perm_identity(uint32_t (*perm)[SETUP_NT], int t) {
    for (int w = 0; w < 64; w++) perm[w][t] = 0x03020100u + 0x04040404u * (uint32_t)w;
}
__device__ __forceinline__ void perm_store(uint32_t (*perm)[SETUP_NT], int t, MgLattice *L) {
    uint4 *dst = reinterpret_cast<uint4 *>(L->p);
#pragma unroll 4
    for (int q = 0; q < 16; q++) dst[q] = make_uint4(perm[4 * q][t], perm[4 * q + 1][t], perm[4 * q + 2][t], perm[4 * q + 3][t]);
}
__device__ __forceinline__ void header_store(MgLattice &h, MgLattice *L, bool dbl) {
    lattice_header(h, dbl);
    const uint4 *src = reinterpret_cast<const uint4 *>(&h);
    uint4 *dst = reinterpret_cast<uint4 *>(L);
#pragma unroll
    for (int q = 0; q < MG_LAT_HDR_WORDS; q++) dst[q] = src[q];
}

/* Overworld: lattice j of seed s; table layout noise-major, then stack, then level
 * (engine/mc_climate.h:95-106, engine/mc_noise.h:255-265). */
__global__ void __launch_bounds__(SETUP_NT) k_setup_xo(const __grid_constant__ MgWorldDesc W, const int64_t *__restrict__ seeds,
                                                       int ns, MgLattice *__restrict__ out) {
    __shared__ uint32_t perm[64][SETUP_NT];
    const int t = threadIdx.x;
    const int nt = W.ntables;
    const long long g = (long long)blockIdx.x * SETUP_NT + t;
    if (g >= (long long)ns * nt) return;
    const int s = (int)(g / nt), j = (int)(g % nt);
    int i = 0;
    while (i < MG_OW_NOISES - 1 && j >= W.noise[i + 1].base) i++;
    const MgNoise &N = W.noise[i];
    const int r = j - N.base, st = r >= N.nlev, k = r - st * N.nlev;
    Xo root = xo_from_seed(seeds[s]);
    uint64_t plo = xo_next(root), phi = xo_next(root);   /* forkPositional */
    Xo nr = xo_make(W.nhl[i] ^ plo, W.nhh[i] ^ phi);      /* fromHashOf("minecraft:<noise>") */
    uint64_t a = xo_next(nr), b = xo_next(nr);            /* first stack's forkPositional */
    if (st) { a = xo_next(nr); b = xo_next(nr); }         /* second stack's */
    Xo x = xo_make(N.hlo[k] ^ a, N.hhi[k] ^ b);           /* fromHashOf("octave_<n>") */
    MgLattice h;
    h.ox = xo_double(x) * 256.0;
    h.oy = xo_double(x) * 256.0;
    h.oz = xo_double(x) * 256.0;
    perm_identity(perm, t);
    xo_shuffle<SETUP_NT>(reinterpret_cast<uint8_t *>(&perm[0][t]), x);
    MgLattice *L = out + g;
    header_store(h, L, !W.fmode);
    perm_store(perm, t, L);
}

/* Nether biome noises: temperature from LCG(seed), vegetation from LCG(seed + 1); LEGACY_GROUP threads per (seed, noise) */
__global__ void __launch_bounds__(SETUP_NT) k_setup_legacy(const __grid_constant__ MgWorldDesc W, const int64_t *__restrict__ seeds,
                                                           int ns, MgLattice *__restrict__ out) {
    __shared__ uint32_t perm[64][SETUP_NT];
    const int t = threadIdx.x;
    const long long g = legacy_index((long long)blockIdx.x * SETUP_NT + t);
    if (g < 0 || g >= 2LL * ns) return;
    const MgNoise &N = W.nether[g & 1];
    MgLattice *T = out + (size_t)(g >> 1) * W.ntables + N.base;
    legacy_noise<SETUP_NT>(N, (int)(g & 1), seeds[g >> 1], &perm[0][t], [&](int i, MgLattice &h) {
        header_store(h, T + i, !W.fmode);
        perm_store(perm, t, T + i);
    });
}
__global__ void __launch_bounds__(SETUP_NT) k_setup_end(const int64_t *__restrict__ seeds, int ns, MgLattice *__restrict__ out) {
    __shared__ uint32_t perm[64][SETUP_NT];
    const int t = threadIdx.x;
    const long long g = (long long)blockIdx.x * SETUP_NT + t;
    if (g >= ns) return;
    MgLattice h;
    legacy_end<SETUP_NT>(seeds[g], &perm[0][t], h);
    header_store(h, out + g, false); /* the End reads the permutation only */
    perm_store(perm, t, out + g);
}

/* ============================================================================ sampling kernels */
/* Stage the seed-independent spline and one seed's lattices in shared memory. */
__device__ __forceinline__ void stage(const MgWorldDesc &W, const MgLattice *__restrict__ src, int n, MgLattice *dstT,
                                      MgSpline *dstS, bool spline) {
    const uint4 *a = reinterpret_cast<const uint4 *>(src);
    uint4 *b = reinterpret_cast<uint4 *>(dstT);
    for (int i = threadIdx.x; i < n * (int)(sizeof(MgLattice) / 16); i += blockDim.x) b[i] = a[i];
    if (spline) {
        const uint4 *c = reinterpret_cast<const uint4 *>(&W.spline);
        uint4 *d = reinterpret_cast<uint4 *>(dstS);
        for (int i = threadIdx.x; i < (int)(sizeof(MgSpline) / 16); i += blockDim.x) d[i] = c[i];
    }
}

/* seeds x points, ENGINE rule.  One thread per sample; lattices of the sample's seed through L1. */
template <bool FM, int DIM>
__global__ void __launch_bounds__(128) k_points(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                const MgLattice *__restrict__ states, int ns,
                                                const int32_t *__restrict__ pts, int np, uint8_t *__restrict__ out,
                                                int32_t *__restrict__ targets) {
    __shared__ MgSpline S;
    if (DIM == MG_OVERWORLD) {
        const uint4 *c = reinterpret_cast<const uint4 *>(&W.spline);
        uint4 *d = reinterpret_cast<uint4 *>(&S);
        for (int i = threadIdx.x; i < (int)(sizeof(MgSpline) / 16); i += blockDim.x) d[i] = c[i];
        __syncthreads();
    }
    long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (DIM == MG_END) g >>= 5; /* a warp per sample */
    if (g >= (long long)ns * np) return;
    const int s = (int)(g / np), p = (int)(g % np);
    const int qx = pts[3 * p], qy = pts[3 * p + 1], qz = pts[3 * p + 2];
    const MgLattice *T = states + (size_t)s * W.ntables;
    int32_t tg[6];
    if (DIM == MG_END) {
        const int c = end_chunk_class(T->p, FM, (qx * 4) >> 4, (qz * 4) >> 4, W.end_f2, W.end_g2);
        if (threadIdx.x & 31) return;
        out[g] = (uint8_t)W.end_ids[c];
        if (targets)
            for (int k = 0; k < 6; k++) targets[g * 6 + k] = 0;
        return;
    }
    cell_target<FM, DIM>(W, S, T, qx, qy, qz, tg);
    uint64_t d;
    int leaf = tree_search_scattered(tree, tg, -1, d);
    out[g] = tree[leaf].biome;
    if (targets)
        for (int k = 0; k < 6; k++) targets[g * 6 + k] = tg[k];
}

/* One seed's quart grid, a thread per cell: the Nether's, and the Overworld's of worlds that the tile kernels do not take
 * (ow_tile_supported).  ENGINE: biome ids.  GRID_CHAIN: first minimum leaf, its fitness, tie flag and
 * the target of every cell, for k_chain_resolve. */
template <bool FM, int DIM, bool CHAIN>
__global__ void __launch_bounds__(128) k_grid(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                              const MgLattice *__restrict__ state, int qx0, int qz0, int nx, int nz,
                                              int qy, uint8_t *__restrict__ out, ChainRec *__restrict__ rec) {
    extern __shared__ uint4 smem_raw[];
    MgSpline *S = reinterpret_cast<MgSpline *>(smem_raw);
    MgLattice *T = reinterpret_cast<MgLattice *>(S + 1);
    stage(W, state, W.ntables, T, S, DIM == MG_OVERWORLD);
    __syncthreads();
    const int tw = mg_parts(nx, 8); /* 8 x 16-cell tiles */
    const int ix = (int)(blockIdx.x % (unsigned)tw) * 8 + threadIdx.x % 8, iz = (int)(blockIdx.x / (unsigned)tw) * 16 + threadIdx.x / 8;
    if (ix >= nx || iz >= nz) return;
    const long long g = (long long)iz * nx + ix;
    int32_t tg[6];
    cell_target<FM, DIM>(W, *S, T, qx0 + ix, qy, qz0 + iz, tg);
    uint64_t d;
    if (CHAIN) {
        bool tied;
        const int leaf = tree_search_tie(tree, tg, d, tied);
        out[g] = tree[leaf].biome;
        ChainRec r;
        for (int k = 0; k < 6; k++) r.tg[k] = tg[k];
        r.d = d;
        r.leaf = leaf;
        r.tie = tied;
        rec[g] = r;
    } else {
        out[g] = tree[tree_search(tree, tg, -1, d)].biome;
    }
}
/* GRID_CHAIN: a tied cell takes the previous cell's leaf when that leaf is also at minimum fitness.
 * Walk back to the nearest untied cell (whose leaf is its own first minimum) and replay forward. */
__global__ void k_chain_resolve(const MgTreeNode *__restrict__ tree, const ChainRec *__restrict__ rec, long long n,
                                uint8_t *__restrict__ out) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n || !rec[g].tie) return;
    long long j = g - 1;
    while (j >= 0 && rec[j].tie) j--;
    int leaf = j >= 0 ? rec[j].leaf : -1;
    for (long long k = j + 1; k <= g; k++) {
        const ChainRec &r = rec[k];
        if (leaf < 0 || node_dist(tree[leaf], r.tg) != r.d) leaf = r.leaf;
    }
    out[g] = tree[leaf].biome;
}

/* CHUNK_ORDER: the chain runs chunk by chunk (chunk rows tz outer, tx inner) and, inside a chunk, over its
 * cells in the grid (z outer, x inner), across chunks: the order of the 26.3 chunk-batched climate
 * (oracle/src/v263/oracle/compat/Compat.java:168-221 in the reference).  order[pos] = cell index. */
__global__ void k_chain_order(int qx0, int qz0, int nx, int nz, int32_t *__restrict__ order) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (long long)nx * nz) return;
    const int qx = qx0 + (int)(g % nx), qz = qz0 + (int)(g / nx);
    const int tx = qx >> 2, tz = qz >> 2;
    const int za = max(tz * 4, qz0), zb = min(tz * 4 + 3, qz0 + nz - 1);
    const int xa = max(tx * 4, qx0), xb = min(tx * 4 + 3, qx0 + nx - 1);
    const long long pos = (long long)(za - qz0) * nx + (long long)(xa - qx0) * (zb - za + 1) +
                          (long long)(qz - za) * (xb - xa + 1) + (qx - xa);
    order[pos] = (int32_t)g;
}
/* the chain replay of k_chain_resolve along order[] */
__global__ void k_chain_resolve_ordered(const MgTreeNode *__restrict__ tree, const ChainRec *__restrict__ rec, long long n,
                                        const int32_t *__restrict__ order, uint8_t *__restrict__ out) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || !rec[order[p]].tie) return;
    long long j = p - 1;
    while (j >= 0 && rec[order[j]].tie) j--;
    int leaf = j >= 0 ? rec[order[j]].leaf : -1;
    for (long long k = j + 1; k <= p; k++) {
        const ChainRec &r = rec[order[k]];
        if (leaf < 0 || node_dist(tree[leaf], r.tg) != r.d) leaf = r.leaf;
    }
    out[order[p]] = tree[leaf].biome;
}

/* (the Nether's, the End's by a table of classes, and the Overworld's of worlds that the tile kernels do not take)
 * mcgen_biome_grid: out[iz*nx+ix] = biome_at(x0 + ix*step, y, z0 + iz*step) (libmcgen/src/region.c:86-108) */
template <bool FM, int DIM>
__global__ void __launch_bounds__(128, 6) k_blockgrid(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                   const MgLattice *__restrict__ state, int64_t zseed, int x0, int z0,
                                                   int nx, int nz, int step, int y, const int32_t *__restrict__ xyz,
                                                   uint8_t *__restrict__ out, const uint8_t *__restrict__ end_cls,
                                                   int ecx0, int ecz0, int encx) {
    extern __shared__ uint4 smem_raw[];
    MgSpline *S = reinterpret_cast<MgSpline *>(smem_raw);
    MgLattice *T = reinterpret_cast<MgLattice *>(S + 1);
    if (DIM != MG_END) {
        stage(W, state, W.ntables, T, S, DIM == MG_OVERWORLD);
        __syncthreads();
    }
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = g < (long long)nx * nz;
    if (!in) return;
    int bxk, byk, bzk;
    if (xyz) { bxk = xyz[3 * g]; byk = xyz[3 * g + 1]; bzk = xyz[3 * g + 2]; }
    else { bxk = x0 + (int)(g % nx) * step; byk = y; bzk = z0 + (int)(g / nx) * step; }
    int cx, cy, cz;
    zoom_cell(zseed, bxk, byk, bzk, cx, cy, cz);
    if (DIM == MG_END) {
        int chx = (cx * 4) >> 4, chz = (cz * 4) >> 4;
        out[g] = (uint8_t)W.end_ids[end_cls[(size_t)(chz - ecz0) * encx + (chx - ecx0)]];
        return;
    }
    out[g] = (uint8_t)cell_chunk<FM, DIM>(W, *S, T, tree, cx, cy, cz);
}
/* Block points, one per warp (wc_*): a point's octaves, zoom candidates and tree nodes over the lanes.  A thread per point ran
 * them in series: one point took 90 us, and a warp of unrelated points diverged in every search. */
template <bool FM, int DIM>
__device__ __forceinline__ void block_points(const MgWorldDesc &W, const MgTreeNode *__restrict__ tree, const MgLattice *__restrict__ state,
                                             int64_t zseed, const int32_t *xyz, int n, uint8_t *__restrict__ out) {
    extern __shared__ uint4 smem_raw[];
    WcStage &st = *reinterpret_cast<WcStage *>(smem_raw);
    wc_stage(st, W, state, threadIdx.x, blockDim.x);
    __syncthreads();
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += (int)((gridDim.x * blockDim.x) >> 5)) {
        int cx, cy, cz;
        wc_zoom(zseed, xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2], cx, cy, cz);
        const int b = wc_cell_chunk<FM, DIM>(W, st.spline, st.lat, tree, cx, cy, cz);
        if ((threadIdx.x & 31) == 0) out[i] = (uint8_t)b;
    }
}
template <bool FM, int DIM>
__global__ void __launch_bounds__(128) k_block_points(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                      const MgLattice *__restrict__ state, int64_t zseed,
                                                      const int32_t *__restrict__ xyz, int n, uint8_t *__restrict__ out) {
    block_points<FM, DIM>(W, tree, state, zseed, xyz, n, out);
}
/* a few points, their coordinates in the launch itself (no buffers, no copies, with the ids
 * stored to pinned host memory: a one-point call 47 -> 36 us in 26.1, 38 -> 30 in 26.3, 34 -> 23 in the Nether) */
struct FewPoints {
    int32_t xyz[3 * FEW_POINTS];
};
template <bool FM, int DIM>
__global__ void __launch_bounds__(128) k_block_few(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                   const MgLattice *__restrict__ state, int64_t zseed, const __grid_constant__ FewPoints p,
                                                   int n, uint8_t *__restrict__ out) {
    block_points<FM, DIM>(W, tree, state, zseed, p.xyz, n, out);
}
/* sparse End samples (a grid, or nx points at xyz), whose chunks are not worth a table of classes: one per warp */
template <bool FM>
__global__ void __launch_bounds__(128) k_end_samples(const __grid_constant__ MgWorldDesc W, const MgLattice *__restrict__ state,
                                                     int64_t zseed, int x0, int z0, int nx, long long n, int step, int y,
                                                     const int32_t *__restrict__ xyz, uint8_t *__restrict__ out) {
    __shared__ uint8_t p[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) p[i] = state->p[i];
    __syncthreads();
    for (long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < n; g += (long long)gridDim.x * blockDim.x >> 5) {
        const int x = xyz ? xyz[3 * g] : x0 + (int)(g % nx) * step, z = xyz ? xyz[3 * g + 2] : z0 + (int)(g / nx) * step;
        int cx, cy, cz;
        zoom_cell(zseed, x, xyz ? xyz[3 * g + 1] : y, z, cx, cy, cz);
        const int c = end_chunk_class(p, FM, (cx * 4) >> 4, (cz * 4) >> 4, W.end_f2, W.end_g2);
        if ((threadIdx.x & 31) == 0) out[g] = (uint8_t)W.end_ids[c];
    }
}
/* End class of chunks [cx0, cx0+ncx) x [cz0, cz0+ncz): one w x h-chunk tile per block (endtile.cuh) */
template <bool FM>
__global__ void __launch_bounds__(128) k_end_chunks(const MgLattice *__restrict__ state, int cx0, int cz0, int ncx,
                                                    int ncz, int w, int h, uint8_t *__restrict__ cls, double F2, double G2) {
    __shared__ uint8_t p[256];
    __shared__ EndTile tile;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) p[i] = state->p[i];
    end_tile_grad(state->p, tile);
    __syncthreads();
    const int tw = (ncx + w - 1) / w;
    const int tx0 = cx0 + (int)(blockIdx.x % tw) * w, tz0 = cz0 + (int)(blockIdx.x / tw) * h;
    end_tile_classes<FM>(p, F2, G2, tx0, tz0, w, h, tile);
    for (int i = threadIdx.x; i < w * h; i += blockDim.x) {
        const int cx = tx0 + i % w, cz = tz0 + i / w;
        if (cx < cx0 + ncx && cz < cz0 + ncz) cls[(size_t)(cz - cz0) * ncx + (cx - cx0)] = tile.cls[i];
    }
}

/* ============================================================================ host launchers */
static inline unsigned blocks_for(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }
/* one grid's classes: large tiles (fewer window cells a chunk) once they fill the chip, else tiles of 8 x 8 */
static void end_chunks(const MgWorldDesc &W, const MgLattice *state, int cx0, int cz0, int ncx, int ncz, uint8_t *cls, cudaStream_t st) {
    const int cap = (long long)ncx * ncz >= 152LL * END_TC * END_TC ? END_TC : 8;
    const int w = end_tile_side(ncx, cap), h = end_tile_side(ncz, cap);
    const unsigned tiles = (unsigned)((long long)((ncx + w - 1) / w) * ((ncz + h - 1) / h));
    ProfScope ps_(K_END_CHUNKS, st);
    if (W.fmode) k_end_chunks<true><<<tiles, 128, 0, st>>>(state, cx0, cz0, ncx, ncz, w, h, cls, W.end_f2, W.end_g2);
    else k_end_chunks<false><<<tiles, 128, 0, st>>>(state, cx0, cz0, ncx, ncz, w, h, cls, W.end_f2, W.end_g2);
    count_launch();
}
static size_t grid_smem(const MgWorldDesc &W) { return sizeof(MgSpline) + (size_t)W.ntables * sizeof(MgLattice); }
int launch_setup(const MgWorldDesc &W, const int64_t *d_seeds, int ns, MgLattice *d_states, cudaStream_t st) {
    if (ns <= 0) return 0;
    if (W.dim == MG_OVERWORLD) {
        long long n = (long long)ns * W.ntables;
        { ProfScope ps_(K_SETUP_XO, st); k_setup_xo<<<blocks_for(n, SETUP_NT), SETUP_NT, 0, st>>>(W, d_seeds, ns, d_states); }
    } else if (W.dim == MG_NETHER) {
        { ProfScope ps_(K_SETUP_LEGACY, st); k_setup_legacy<<<blocks_for(legacy_threads(2LL * ns), SETUP_NT), SETUP_NT, 0, st>>>(W, d_seeds, ns, d_states); }
    } else {
        { ProfScope ps_(K_SETUP_END, st); k_setup_end<<<blocks_for(ns, SETUP_NT), SETUP_NT, 0, st>>>(d_seeds, ns, d_states); }
    }
    count_launch();
    return (int)cudaGetLastError();
}

/* Overworld density functions at block points (x, y, z): out[5 i + k] = continents, erosion, ridges, offset,
 * depth as the climate sampler computes them before it rounds them to floats (engine/mc_climate.h:113-164 at
 * block coordinates; the reference Java oracle's "df" values, oracle/gen_vectors.py:76-84).  Double branch:
 * every noise by the exact double evaluation (no screen: the doubles themselves are the result); float
 * branch: the floats, widened.  One thread per point, one seed's lattices through L1. */
template <bool FM>
__global__ void __launch_bounds__(128) k_density(const __grid_constant__ MgWorldDesc W, const MgLattice *__restrict__ T,
                                                 int n, const int32_t *__restrict__ xyz, double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int bx = xyz[3 * i], by = xyz[3 * i + 1], bz = xyz[3 * i + 2];
    const double X = bx * 0.25, Z = bz * 0.25, Xc = X * MG_SECOND_STACK, Zc = Z * MG_SECOND_STACK;
    double v[5];
    if (FM) {
        const float sx = nn_f_y0(W.noise[0], T, X, Z, Xc, Zc) * 4.0f; /* ShiftA (x, 0, z) */
        const float sz = nn_f_z0(W.noise[0], T, Z, X, Zc, Xc) * 4.0f; /* ShiftB (z, x, 0) */
        const double x = X + (double)sx, z = Z + (double)sz, xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
        const float c = nn_f_y0(W.noise[3], T, x, z, xc, zc);
        const float e = nn_f_y0(W.noise[4], T, x, z, xc, zc);
        const float r = nn_f_y0(W.noise[5], T, x, z, xc, zc);
        const float a = fabsf(r) + W.rf_f[0];
        const float co[4] = {c, e, r, (fabsf(a) + W.rf_f[1]) * W.rf_f[2]};
        const float off = W.off_f + spline_eval(W.spline, co);
        const int lo = min(W.grad_from_y, W.grad_to_y), hi = max(W.grad_from_y, W.grad_to_y);
        const int yy = by < lo ? lo : (by > hi ? hi : by);
        const float depth = (W.grad_from_f + (float)(yy - W.grad_from_y) * W.grad_fac_f) + off;
        v[0] = c; v[1] = e; v[2] = r; v[3] = off; v[4] = depth;
    } else {
        const double x = X + nn_d_y0(W.noise[0], T, X, Z, Xc, Zc) * 4.0;
        const double z = Z + nn_d_z0(W.noise[0], T, Z, X, Zc, Xc) * 4.0;
        const double xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
        const double c = nn_d_y0(W.noise[3], T, x, z, xc, zc);
        const double e = nn_d_y0(W.noise[4], T, x, z, xc, zc);
        const double r = nn_d_y0(W.noise[5], T, x, z, xc, zc);
        const float co[4] = {(float)c, (float)e, (float)r, (float)ridges_folded_d(W, r)};
        const double off = 0.0 + (W.off_d + (double)spline_eval(W.spline, co)) * 1.0;
        v[0] = c; v[1] = e; v[2] = r; v[3] = off; v[4] = depth_grad_d(W, by) + off;
    }
    for (int k = 0; k < 5; k++) out[5 * (size_t)i + k] = v[k];
}

template <bool FM, int DIM>
static void points_t(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *states, int ns, const int32_t *pts,
                     int np, uint8_t *out, int32_t *tg, cudaStream_t st) {
    long long n = (long long)ns * np;
    { ProfScope ps_(K_POINTS, st); k_points<FM, DIM><<<blocks_for(DIM == MG_END ? 32 * n : n, 128), 128, 0, st>>>(W, tree, states, ns, pts, np, out, tg); }
}
int launch_points(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *states, int ns, const int32_t *pts,
                  int np, uint8_t *out, int32_t *tg, cudaStream_t st) {
    if ((long long)ns * np <= 0) return 0;
    if (W.fmode) {
        if (W.dim == MG_OVERWORLD) points_t<true, MG_OVERWORLD>(W, tree, states, ns, pts, np, out, tg, st);
        else if (W.dim == MG_NETHER) points_t<true, MG_NETHER>(W, tree, states, ns, pts, np, out, tg, st);
        else points_t<true, MG_END>(W, tree, states, ns, pts, np, out, tg, st);
    } else {
        if (W.dim == MG_OVERWORLD) points_t<false, MG_OVERWORLD>(W, tree, states, ns, pts, np, out, tg, st);
        else if (W.dim == MG_NETHER) points_t<false, MG_NETHER>(W, tree, states, ns, pts, np, out, tg, st);
        else points_t<false, MG_END>(W, tree, states, ns, pts, np, out, tg, st);
    }
    count_launch();
    return (int)cudaGetLastError();
}

int launch_density(const MgWorldDesc &W, const MgLattice *state, int n, const int32_t *xyz, double *out, cudaStream_t st) {
    if (n <= 0) return 0;
    if (W.dim != MG_OVERWORLD) return (int)cudaErrorInvalidValue;
    {
        ProfScope ps_(K_DENSITY, st);
        if (W.fmode) k_density<true><<<blocks_for(n, 128), 128, 0, st>>>(W, state, n, xyz, out);
        else k_density<false><<<blocks_for(n, 128), 128, 0, st>>>(W, state, n, xyz, out);
    }
    count_launch();
    return (int)cudaGetLastError();
}

template <bool FM, int DIM, bool CHAIN>
static void grid_t(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *state, int qx0, int qz0, int nx, int nz,
                   int qy, uint8_t *out, ChainRec *rec, cudaStream_t st) {
    size_t sm = grid_smem(W);
    cudaFuncSetAttribute(k_grid<FM, DIM, CHAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const long long tiles = (long long)mg_parts(nx, 8) * mg_parts(nz, 16);
    { ProfScope ps_(K_GRID, st); k_grid<FM, DIM, CHAIN><<<(unsigned)tiles, 128, sm, st>>>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec); }
    count_launch();
}
__global__ void k_end_lookup(const __grid_constant__ MgWorldDesc W, const uint8_t *__restrict__ cls, int cx0, int cz0,
                             int ncx, int qx0, int qz0, int nx, int nz, uint8_t *__restrict__ out) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (long long)nx * nz) return;
    int qx = qx0 + (int)(g % nx), qz = qz0 + (int)(g / nx);
    int cx = (qx * 4) >> 4, cz = (qz * 4) >> 4;
    out[g] = (uint8_t)W.end_ids[cls[(size_t)(cz - cz0) * ncx + (cx - cx0)]];
}
int launch_end_lookup(const MgWorldDesc &W, const uint8_t *cls, int cx0, int cz0, int ncx, int qx0, int qz0, int nx,
                      int nz, uint8_t *out, cudaStream_t st) {
    { ProfScope ps_(K_END_LOOKUP, st); k_end_lookup<<<blocks_for((long long)nx * nz, 256), 256, 0, st>>>(W, cls, cx0, cz0, ncx, qx0, qz0, nx, nz, out); }
    count_launch();
    return (int)cudaGetLastError();
}
/* chain records, then their order; (Overworld) the tile kernels' scratch takes the order's place, which is written later, or where
 * the grid is too small for that follows it */
static size_t order_bytes(long long n) { return (size_t)n * sizeof(int32_t); }
static size_t chain_bytes(long long n) { return ((size_t)n * sizeof(ChainRec) + order_bytes(n) + 15) & ~(size_t)15; }
static bool chain_rule(int rule) { return rule == MG_TIE_GRID_CHAIN || rule == MG_TIE_CHUNK_ORDER; }
size_t quart_scratch_bytes(const MgWorldDesc &W, int rule, int nx, int nz) {
    if (W.dim == MG_END) return (size_t)(nx / 4 + 3) * (size_t)(nz / 4 + 3);
    const long long n = (long long)nx * nz;
    const size_t tiles = ow_tile_supported(W) ? ow_grid_scratch_bytes(W, false, n) : 0;
    return chain_rule(rule) ? chain_bytes(n) + (tiles > order_bytes(n) ? tiles : 0) : tiles;
}
int launch_quart_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int qx0, int qz0,
                      int nx, int nz, int qy, int rule, uint8_t *out, void *scratch, cudaStream_t st) {
    long long n = (long long)nx * nz;
    if (n <= 0) return 0;
    if (W.dim == MG_END) {
        /* chunk classes over the grid's chunk range, then one lookup per cell */
        int cx0 = (qx0 * 4) >> 4, cz0 = (qz0 * 4) >> 4;
        int cx1 = ((qx0 + nx - 1) * 4) >> 4, cz1 = ((qz0 + nz - 1) * 4) >> 4;
        int ncx = cx1 - cx0 + 1, ncz = cz1 - cz0 + 1;
        uint8_t *cls = (uint8_t *)scratch;
        end_chunks(W, state, cx0, cz0, ncx, ncz, cls, st);
        return launch_end_lookup(W, cls, cx0, cz0, ncx, qx0, qz0, nx, nz, out, st);
    }
    const bool chain = chain_rule(rule);
    ChainRec *rec = (ChainRec *)scratch;
    if (ow_tile_supported(W) && !ow_beyond(W.fmode != 0, OT_FEW_CELLS, qx0, qz0, (long long)qx0 + nx - 1, (long long)qz0 + nz - 1, n)) {
        const size_t tiles = ow_grid_scratch_bytes(W, false, n);
        uint8_t *more = !tiles ? nullptr : !chain ? (uint8_t *)scratch : (uint8_t *)scratch + (tiles > order_bytes(n) ? chain_bytes(n) : sizeof(ChainRec) * (size_t)n);
        const int rows = (int)(0x7FFFFFFF / nx); /* cell indices of a tile grid are 32-bit */
        for (int z = 0; z < nz; z += rows) {
            const size_t at = (size_t)z * (size_t)nx;
            const int rc = launch_ow_quart_grid(W, d_world, tree, state, qx0, qz0 + z, nx, rows < nz - z ? rows : nz - z, qy,
                                                chain ? rec + at : nullptr, out + at, more, st);
            if (rc) return rc;
            if (rows >= nz - z) break;
        }
    } else if (W.fmode) {
        if (W.dim == MG_OVERWORLD) {
            if (chain) grid_t<true, MG_OVERWORLD, true>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
            else grid_t<true, MG_OVERWORLD, false>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
        } else {
            if (chain) grid_t<true, MG_NETHER, true>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
            else grid_t<true, MG_NETHER, false>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
        }
    } else {
        if (W.dim == MG_OVERWORLD) {
            if (chain) grid_t<false, MG_OVERWORLD, true>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
            else grid_t<false, MG_OVERWORLD, false>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
        } else {
            if (chain) grid_t<false, MG_NETHER, true>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
            else grid_t<false, MG_NETHER, false>(W, tree, state, qx0, qz0, nx, nz, qy, out, rec, st);
        }
    }
    if (rule == MG_TIE_GRID_CHAIN) {
        { ProfScope ps_(K_CHAIN_RESOLVE, st); k_chain_resolve<<<blocks_for(n, 256), 256, 0, st>>>(tree, rec, n, out); }
        count_launch();
    } else if (rule == MG_TIE_CHUNK_ORDER) {
        int32_t *order = reinterpret_cast<int32_t *>(rec + n);
        { ProfScope ps_(K_CHAIN_RESOLVE, st); k_chain_order<<<blocks_for(n, 256), 256, 0, st>>>(qx0, qz0, nx, nz, order); }
        count_launch();
        { ProfScope ps_(K_CHAIN_RESOLVE, st); k_chain_resolve_ordered<<<blocks_for(n, 256), 256, 0, st>>>(tree, rec, n, order, out); }
        count_launch();
    }
    return (int)cudaGetLastError();
}

template <bool FM, int DIM>
static void blockgrid_t(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *state, int64_t zseed, int x0,
                        int z0, int nx, int nz, int step, int y, const int32_t *xyz, uint8_t *out, const uint8_t *cls,
                        int ecx0, int ecz0, int encx, cudaStream_t st) {
    size_t sm = DIM == MG_END ? 0 : grid_smem(W);
    ProfScope ps_(K_BLOCKGRID, st);
    if (DIM == MG_END && !cls) {
        const long long n = (long long)nx * nz, nb = (n + 3) / 4;
        k_end_samples<FM><<<(unsigned)(nb < 16 * 152 ? nb : 16 * 152), 128, 0, st>>>(W, state, zseed, x0, z0, nx, n, step, y, xyz, out);
        return;
    }
    if constexpr (DIM != MG_END) {
        /* the Nether's cells are cheap enough for a thread each once there are enough of them (26.1: 3,000 points 19.8 us by warps,
         * 22.0 by threads; 14,108 points 67.6 and 30.5) */
        const bool lanes = DIM == MG_OVERWORLD ? W.noise[0].nlev <= 8 : W.ntables <= 32; /* wc_target's lists */
        if (xyz && lanes && (DIM == MG_OVERWORLD || nx <= 3072)) {
            const long long nb = ((long long)nx + 3) / 4;
            k_block_points<FM, DIM><<<(unsigned)(nb < 16 * 152 ? nb : 16 * 152), 128, sizeof(WcStage), st>>>(W, tree, state, zseed, xyz, nx,
                                                                                                          out);
            return;
        }
    }
    if (sm) cudaFuncSetAttribute(k_blockgrid<FM, DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const unsigned nb = blocks_for((long long)nx * nz, 128);
    k_blockgrid<FM, DIM><<<nb, 128, sm, st>>>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0,
                                              encx);
}
/* the scratch holds only the record of open cells, and without it (null) those are evaluated where they occur */
bool quart_scratch_optional(const MgWorldDesc &W, int rule) { return W.dim == MG_OVERWORLD && !chain_rule(rule); }
/* maps, and lists of so many points that a thread each (k_ow_sparse, 140 to 180 us for the first) is faster than a warp each: 26.1
 * 6,000 points 153 against 138 us, 10,000 161 and 204, 400,000 2,070 and 5,694; 26.3 20,000 points 188 and 180, 100,000 327 and 637 */
static bool block_tiles(const MgWorldDesc &W, int x0, int z0, int nx, bool points) {
    return ow_block_grid_supported(W, x0, z0) && (!points || nx > (W.fmode ? 24576 : 8192));
}
size_t block_scratch_bytes(const MgWorldDesc &W, int x0, int z0, int nx, int nz, bool points) {
    return W.dim == MG_OVERWORLD && block_tiles(W, x0, z0, nx, points) ? ow_grid_scratch_bytes(W, true, (long long)nx * nz) : 0;
}
bool block_few_supported(const MgWorldDesc &W, int n) {
    return n <= FEW_POINTS && (W.dim == MG_OVERWORLD ? W.noise[0].nlev <= 8 : W.dim == MG_NETHER && W.ntables <= 32);
}
template <bool FM, int DIM>
static void few_t(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *state, int64_t zseed, const FewPoints &p, int n,
                  uint8_t *out, cudaStream_t st) {
    ProfScope ps_(K_BLOCKGRID, st);
    k_block_few<FM, DIM><<<(unsigned)((n + 3) / 4), 128, sizeof(WcStage), st>>>(W, tree, state, zseed, p, n, out);
}
int launch_block_few(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *state, int64_t zseed, const int32_t *xyz, int n,
                     uint8_t *out, cudaStream_t st) {
    FewPoints p = {};
    memcpy(p.xyz, xyz, sizeof(int32_t) * 3 * (size_t)n);
    if (W.dim == MG_OVERWORLD) {
        if (W.fmode) few_t<true, MG_OVERWORLD>(W, tree, state, zseed, p, n, out, st);
        else few_t<false, MG_OVERWORLD>(W, tree, state, zseed, p, n, out, st);
    } else {
        if (W.fmode) few_t<true, MG_NETHER>(W, tree, state, zseed, p, n, out, st);
        else few_t<false, MG_NETHER>(W, tree, state, zseed, p, n, out, st);
    }
    count_launch();
    return (int)cudaGetLastError();
}
/* Block-coordinate biomes: a grid (xyz == nullptr) or n = nx points (nz == 1) at xyz. For the End,
 * `scratch` holds the chunk classes of [ecx0, ecx0+encx) x [ecz0, ecz0+encz). */
int launch_block_biomes(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int64_t zseed,
                        int x0, int z0, int nx, int nz, int step, int y, const int32_t *xyz, uint8_t *out, void *scratch,
                        int ecx0, int ecz0, int encx, int encz, cudaStream_t st) {
    if ((long long)nx * nz <= 0) return 0;
    if (W.dim == MG_OVERWORLD && block_tiles(W, x0, z0, nx, xyz != nullptr))
        return launch_ow_block_grid(W, d_world, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, scratch, st);
    uint8_t *cls = (uint8_t *)scratch; /* End chunk classes, or null: evaluate per sample */
    if (W.dim == MG_END && cls) {
        end_chunks(W, state, ecx0, ecz0, encx, encz, cls, st);
    }
    if (W.fmode) {
        if (W.dim == MG_OVERWORLD) blockgrid_t<true, MG_OVERWORLD>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
        else if (W.dim == MG_NETHER) blockgrid_t<true, MG_NETHER>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
        else blockgrid_t<true, MG_END>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
    } else {
        if (W.dim == MG_OVERWORLD) blockgrid_t<false, MG_OVERWORLD>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
        else if (W.dim == MG_NETHER) blockgrid_t<false, MG_NETHER>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
        else blockgrid_t<false, MG_END>(W, tree, state, zseed, x0, z0, nx, nz, step, y, xyz, out, cls, ecx0, ecz0, encx, st);
    }
    count_launch();
    return (int)cudaGetLastError();
}

}  // namespace mg
