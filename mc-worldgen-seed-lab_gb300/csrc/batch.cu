/* batch.cu -- many biome-map requests of uneven size in a few persistent launches: the Overworld's go to the tile kernels of
 * owtile.cu, one per branch, everything else to k_batch here.
 *
 * A request is (world: version + dimension + preset, seed, quart region qx0..qx0+nx-1 x qz0..qz0+nz-1 at
 * quart y, tie rule).  The host splits every request into tiles -- 32 x 32 cells for the Nether (nethertile.cuh), equal parts of
 * up to 24 x 24 chunks for the End (endtile.cuh), 128 cells (8 x 16) for what has no tile form (worlds with other noises than the
 * game's; the double branch's Overworld beyond the tables' coordinates) --
 * and numbers them.  k_batch runs as many CTAs as fit for the whole batch; each CTA takes the next tile
 * from a device counter (the work queue), finds its request among the requests' first-tile numbers, stages
 * that request's seed lattices in shared memory when they differ from the previous tile's, and computes the
 * tile.  Uneven requests therefore cost no idle SMs and no per-request launches.
 *
 * The seed lattices of every (world, seed) of the batch are built beforehand by k_setup_list_* into a
 * state pool (the served form keeps that pool across batches as a device cache).  All these kernels overlap (overlap.cuh).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "batch.h"
#include "batchdev.cuh"
#include "climate.cuh"
#include "endtile.cuh"
#include "launch.h"
#include "legacy.cuh"
#include "nethertile.cuh"
#include "overlap.cuh"
#include "prof.h"

namespace mg {

#define BNT 128        /* threads per CTA */

/* ---------------------------------------------------------------- setup of a list of (world, seed) */
#define LNT 128
__device__ __forceinline__ void lst_store(uint32_t (*perm)[LNT], int t, MgLattice &h, MgLattice *L, bool dbl) {
    lattice_header(h, dbl);
    const uint4 *src = reinterpret_cast<const uint4 *>(&h);
    uint4 *dst = reinterpret_cast<uint4 *>(L);
    for (int q = 0; q < MG_LAT_HDR_WORDS; q++) dst[q] = src[q];
    uint4 *dp = reinterpret_cast<uint4 *>(L->p);
    for (int q = 0; q < 16; q++) dp[q] = make_uint4(perm[4 * q][t], perm[4 * q + 1][t], perm[4 * q + 2][t], perm[4 * q + 3][t]);
}
/* Overworld entries: one thread per (entry, lattice). */
__global__ void __launch_bounds__(LNT) k_setup_list_xo(const MgWorldDesc *__restrict__ worlds, const MgSetupEntry *__restrict__ ent,
                                                       int n, const int *__restrict__ first_lattice, long long total,
                                                       MgLattice *__restrict__ pool) {
    __shared__ uint32_t perm[64][LNT];
    const int t = threadIdx.x;
    const long long g = (long long)blockIdx.x * LNT + t;
    overlap_next();
    if (g >= total) return;
    int lo = 0, hi = n - 1; /* entry e with first_lattice[e] <= g < first_lattice[e+1] */
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (first_lattice[mid] <= g) lo = mid; else hi = mid - 1;
    }
    const MgSetupEntry &E = ent[lo];
    const MgWorldDesc &W = worlds[E.world];
    const int j = (int)(g - first_lattice[lo]);
    int i = 0;
    while (i < MG_OW_NOISES - 1 && j >= W.noise[i + 1].base) i++;
    const MgNoise &N = W.noise[i];
    const int r = j - N.base, st = r >= N.nlev, k = r - st * N.nlev;
    Xo root = xo_from_seed(E.seed);
    uint64_t plo = xo_next(root), phi = xo_next(root);
    Xo nr = xo_make(W.nhl[i] ^ plo, W.nhh[i] ^ phi);
    uint64_t a = xo_next(nr), b = xo_next(nr);
    if (st) { a = xo_next(nr); b = xo_next(nr); }
    Xo x = xo_make(N.hlo[k] ^ a, N.hhi[k] ^ b);
    MgLattice h;
    h.ox = xo_double(x) * 256.0;
    h.oy = xo_double(x) * 256.0;
    h.oz = xo_double(x) * 256.0;
    for (int w = 0; w < 64; w++) perm[w][t] = 0x03020100u + 0x04040404u * (uint32_t)w;
    uint8_t *mine = reinterpret_cast<uint8_t *>(&perm[0][t]);
    xo_shuffle<LNT>(mine, x);
    lst_store(perm, t, h, pool + E.slot + j, !W.fmode);
    overlap_wait();
}
/* Nether entries: LEGACY_GROUP threads per (entry, noise); End entries: one thread per entry. */
__global__ void __launch_bounds__(LNT) k_setup_list_legacy(const MgWorldDesc *__restrict__ worlds, const MgSetupEntry *__restrict__ ent, int n,
                                                           MgLattice *__restrict__ pool) {
    __shared__ uint32_t perm[64][LNT];
    const int t = threadIdx.x;
    const long long g = legacy_index((long long)blockIdx.x * LNT + t);
    overlap_next();
    if (g < 0 || g >= 2LL * n) return;
    const MgSetupEntry &E = ent[g >> 1];
    const MgWorldDesc &W = worlds[E.world];
    const MgNoise &N = W.nether[g & 1];
    MgLattice *T = pool + E.slot + N.base;
    legacy_noise<LNT>(N, (int)(g & 1), E.seed, &perm[0][t], [&](int i, MgLattice &h) { lst_store(perm, t, h, T + i, !W.fmode); });
    overlap_wait();
}
__global__ void __launch_bounds__(LNT) k_setup_list_end(const MgSetupEntry *__restrict__ ent, int n, MgLattice *__restrict__ pool) {
    __shared__ uint32_t perm[64][LNT];
    const int t = threadIdx.x;
    const long long g = (long long)blockIdx.x * LNT + t;
    overlap_next();
    if (g >= n) return;
    MgLattice h;
    legacy_end<LNT>(ent[g].seed, &perm[0][t], h);
    lst_store(perm, t, h, pool + ent[g].slot, false); /* the End reads the permutation only */
    overlap_wait();
}

/* ---------------------------------------------------------------- the persistent batch kernel */
/* A request's lattices, the Nether's tables and the End's scratch are never live in the same tile, so they share
 * storage: 17 KB per CTA, which leaves the register budget as the occupancy limit (up to 9 CTAs per SM). */
struct BatchEnd {
    uint8_t endp[256];
    EndTile tile;
};
struct BatchSmem {
    union {
        MgLattice lat[MG_MAX_TABLES];
        BatchEnd end;
        NetherTile nether;
    };
    int tile, req, state;
};

/* The cells of an Overworld or Nether tile.  Each code path's cells (and the End's tiles, batch_end) are a function of their
 * own, out of line: the persistent kernel is then a dispatcher, and each path's registers are allocated for that path
 * alone. */
template <bool FM, int DIM, int TILE_W>
__device__ __noinline__ void batch_cells(const MgWorldDesc &W, const MgSpline &S, const MgLattice *T, const MgTreeNode *tree,
                                         const MgBatchReq &R, int tx0, int tz0, uint8_t *out) {
    const int col = threadIdx.x % TILE_W, row = threadIdx.x / TILE_W;
    const int ix = tx0 + col, iz = tz0 + row;
    if (ix >= R.nx || iz >= R.nz) return;
    const int qx = R.qx0 + ix, qz = R.qz0 + iz;
    int b;
    if (R.tie == MG_TIE_CHUNK_CELL) { /* the request's rule: the same for the whole CTA */
        b = cell_chunk<FM, DIM>(W, S, T, tree, qx, R.qy, qz);
    } else {
        int32_t tg[6];
        cell_target<FM, DIM>(W, S, T, qx, R.qy, qz, tg);
        uint64_t d;
        b = tree[tree_search(tree, tg, -1, d)].biome;
    }
    put_id(out + R.out_off + (size_t)iz * R.nx + ix, b);
}

/* End tile t of a request (tiles counted from the chunk of its first cell): the classes of its chunks, then the request's cells
 * in them */
template <bool FM>
__device__ __noinline__ void batch_end(const MgWorldDesc &W, BatchSmem &sm, const MgBatchReq &R, int t, uint8_t *out) {
    const int c0 = R.qx0 >> 2, d0 = R.qz0 >> 2, ncx = ((R.qx0 + R.nx - 1) >> 2) - c0 + 1, ncz = ((R.qz0 + R.nz - 1) >> 2) - d0 + 1;
    const int w = end_tile_side(ncx, END_TC), h = end_tile_side(ncz, END_TC), tw = (ncx + w - 1) / w;
    const int cx0 = c0 + t % tw * w, cz0 = d0 + t / tw * h;
    /* the request's columns and rows in the tile's chunks (in 64 bits: a tile may end beyond the last one) */
    const long long bx = 4LL * cx0 - R.qx0, bz = 4LL * cz0 - R.qz0;
    const int ix0 = (int)max(bx, 0LL), ix1 = (int)min(bx + 4 * w, (long long)R.nx);
    const int iz0 = (int)max(bz, 0LL), iz1 = (int)min(bz + 4 * h, (long long)R.nz);
    end_tile_classes<FM>(sm.end.endp, W.end_f2, W.end_g2, cx0, cz0, w, h, sm.end.tile);
    for (int r = (int)(threadIdx.x >> 5); r < iz1 - iz0; r += BNT / 32)
        for (int c = (int)(threadIdx.x & 31); c < ix1 - ix0; c += 32) {
            const int ix = ix0 + c, iz = iz0 + r;
            put_id(out + R.out_off + (size_t)iz * R.nx + ix,
                   W.end_ids[sm.end.tile.cls[(((R.qz0 + iz) >> 2) - cz0) * w + ((R.qx0 + ix) >> 2) - cx0]]);
        }
}

/* TILE_W: tile width in cells (tiles are 128 cells); MINB: resident CTAs per SM the register allocation
 * is sized for (6: 80 registers, 7: 72, 8: 64, 9: 56) */
template <int TILE_W, int MINB>
__global__ void __launch_bounds__(BNT, MINB) k_batch(const MgWorldDesc *__restrict__ worlds, const MgTreeNode *const *__restrict__ trees,
                                               const MgBatchReq *__restrict__ reqs, int nreq, long long ntiles,
                                               const MgLattice *__restrict__ pool, unsigned long long *__restrict__ counter,
                                               uint8_t *__restrict__ out) {
    extern __shared__ uint4 smem_raw[];
    BatchSmem &sm = *reinterpret_cast<BatchSmem *>(smem_raw);
    overlap_next();
    if (threadIdx.x == 0) sm.state = -1;
    for (;;) {
        __syncthreads();
        if (threadIdx.x < 32) { /* warp 0 takes the next tile and finds its request */
            long long tile = 0;
            if (threadIdx.x == 0) tile = (long long)atomicAdd(counter, 1ULL);
            tile = __shfl_sync(0xFFFFFFFFu, tile, 0);
            const int r = tile < ntiles ? find_req(reqs, nreq, tile) : -1;
            if (threadIdx.x == 0) {
                sm.tile = (int)(r >= 0 ? tile - reqs[r].tile0 : -1);
                sm.req = r;
            }
        }
        __syncthreads();
        const int r = sm.req;
        if (r < 0) break;
        const MgBatchReq R = reqs[r];
        const MgWorldDesc &W = worlds[R.world];
        /* stage the request's lattices when they change (the world's offset spline, about 11 nodes read per
         * sample, is read in place through L1: kept out of shared memory, it leaves room for 9 CTAs per SM) */
        const bool new_state = R.state != sm.state;
        if (new_state) {
            if (W.dim == MG_END) {
                for (int i = threadIdx.x; i < 256; i += BNT) sm.end.endp[i] = pool[R.state].p[i];
                end_tile_grad(pool[R.state].p, sm.end.tile);
            } else if (nether_tile_supported(W)) {
                nether_stage(W, pool + R.state, trees[R.world], sm.nether);
            } else {
                const uint4 *a = reinterpret_cast<const uint4 *>(pool + R.state);
                uint4 *b = reinterpret_cast<uint4 *>(sm.lat);
                for (int i = threadIdx.x; i < W.ntables * (int)(sizeof(MgLattice) / 16); i += BNT) b[i] = a[i];
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) sm.state = R.state;
        const int tile = sm.tile;
        if (W.dim == MG_END) {
            if (W.fmode) batch_end<true>(W, sm, R, tile, out);
            else batch_end<false>(W, sm, R, tile, out);
            continue;
        }
        if (nether_tile_supported(W)) {
            const int tw = mg_parts(R.nx, NT_W);
            if (W.fmode) nether_tile<true>(W, sm.nether, trees[R.world], R, tile % tw * NT_W, tile / tw * NT_W, out);
            else nether_tile<false>(W, sm.nether, trees[R.world], R, tile % tw * NT_W, tile / tw * NT_W, out);
            continue;
        }
        constexpr int TILE_H = BNT / TILE_W;
        const int tw = mg_parts(R.nx, TILE_W);
        const int tx0 = (tile % tw) * TILE_W, tz0 = (tile / tw) * TILE_H;
        const MgTreeNode *tree = trees[R.world];
        if (W.fmode) {
            if (W.dim == MG_OVERWORLD) batch_cells<true, MG_OVERWORLD, TILE_W>(W, W.spline, sm.lat, tree, R, tx0, tz0, out);
            else batch_cells<true, MG_NETHER, TILE_W>(W, W.spline, sm.lat, tree, R, tx0, tz0, out);
        } else if (W.dim == MG_OVERWORLD) {
            batch_cells<false, MG_OVERWORLD, TILE_W>(W, W.spline, sm.lat, tree, R, tx0, tz0, out);
        } else {
            batch_cells<false, MG_NETHER, TILE_W>(W, W.spline, sm.lat, tree, R, tx0, tz0, out);
        }
    }
    overlap_wait();
}

/* ---------------------------------------------------------------- host side */
/* tile shapes the autotuner chooses from: tile width, and the register budget (resident CTAs per SM: 9, 7,
 * 6, 8) in k_batch's second template argument */
const int kBatchTileWidths[BATCH_SHAPES] = {8, 8, 8, 8};
static int g_resident[BATCH_SHAPES] = {0, 0, 0, 0}; /* CTAs per SM x SMs, per shape (batch_prepare) */

int batch_world_group(const MgWorldDesc &W, int tie) {
    if ((tie != MG_TIE_ENGINE && tie != MG_TIE_CHUNK_CELL) || !ow_tile_supported(W)) return BATCH_REST;
    return W.fmode ? BATCH_OW_F : BATCH_OW_D;
}
int batch_group(int world_group, int qx0, int qz0, int nx, int nz) {
    if (world_group != BATCH_OW_D) return world_group;
    return ow_beyond(false, 0, qx0, qz0, (long long)qx0 + nx - 1, (long long)qz0 + nz - 1, (long long)nx * nz) ? BATCH_REST : world_group;
}

long long batch_tiles(int group, const MgWorldDesc &W, int qx0, int qz0, int nx, int nz, int shape) {
    if (group != BATCH_REST) return ow_tiles(nx, nz);
    if (W.dim == MG_END) {
        const long long ncx = ((qx0 + nx - 1) >> 2) - (qx0 >> 2) + 1, ncz = ((qz0 + nz - 1) >> 2) - (qz0 >> 2) + 1;
        const int w = end_tile_side((int)ncx, END_TC), h = end_tile_side((int)ncz, END_TC);
        return ((ncx + w - 1) / w) * ((ncz + h - 1) / h);
    }
    if (nether_tile_supported(W)) return (long long)mg_parts(nx, NT_W) * mg_parts(nz, NT_W);
    const int tw = kBatchTileWidths[shape], th = BNT / tw;
    return (long long)mg_parts(nx, tw) * mg_parts(nz, th);
}

int launch_setup_list(const MgWorldDesc *d_worlds, int dim, const MgSetupEntry *d_ent, int n, const int *d_first,
                      long long total_lattices, MgLattice *d_pool, bool overlap, cudaStream_t st) {
    if (n <= 0) return 0;
    if (dim == MG_OVERWORLD) {
        ProfScope ps_(K_SETUP_XO, st);
        launch_on(overlap, k_setup_list_xo, (unsigned)((total_lattices + LNT - 1) / LNT), LNT, 0, st, d_worlds, d_ent, n, d_first, total_lattices, d_pool);
    } else if (dim == MG_NETHER) {
        ProfScope ps_(K_SETUP_LEGACY, st);
        launch_on(overlap, k_setup_list_legacy, (unsigned)((legacy_threads(2LL * n) + LNT - 1) / LNT), LNT, 0, st, d_worlds, d_ent, n, d_pool);
    } else {
        ProfScope ps_(K_SETUP_END, st);
        launch_on(overlap, k_setup_list_end, (unsigned)((n + LNT - 1) / LNT), LNT, 0, st, d_ent, n, d_pool);
    }
    count_launch_external();
    return (int)cudaGetLastError();
}

template <int TW, int MB>
static int prepare_t(int shape, int sms) {
    int rc = (int)cudaFuncSetAttribute(k_batch<TW, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BatchSmem));
    int n = 0;
    if (!rc) rc = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_batch<TW, MB>, BNT, sizeof(BatchSmem));
    g_resident[shape] = (n > 0 ? n : 1) * sms;
    return rc;
}
/* kernel attributes (before any capture) and resident CTAs per SM of shape 0 */
int batch_prepare(int *ctas_per_sm) {
    static int prepared_dev = -1; /* the attributes are per device and set once (callers hold the ABI lock) */
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (prepared_dev == dev) {
        if (ctas_per_sm) *ctas_per_sm = g_resident[0] / (sms > 0 ? sms : 1);
        return 0;
    }
    int rc = prepare_t<8, 9>(0, sms);
    if (!rc) rc = prepare_t<8, 7>(1, sms);
    if (!rc) rc = prepare_t<8, 6>(2, sms);
    if (!rc) rc = prepare_t<8, 8>(3, sms);
    if (!rc) rc = ow_prepare();
    if (!rc) prepared_dev = dev;
    if (ctas_per_sm) *ctas_per_sm = g_resident[0] / (sms > 0 ? sms : 1);
    return rc;
}

void batch_open_cap(const long long cells[2], int tie, long long open_cap[2]) {
    open_cap[0] = ow_open_cap(cells[0]);
    open_cap[1] = tie == MG_TIE_CHUNK_CELL ? ow_open_cap(cells[1]) : 0; /* the float branch leaves tied cells only */
}
int launch_batch(const MgWorldDesc *d_worlds, const MgTreeNode *const *d_trees, const MgBatchReq *d_reqs,
                 const BatchGroups &g, int tie, const MgLattice *d_pool, unsigned long long *d_counter, MgOpenCell *d_open,
                 const long long open_cap[2], uint8_t *d_out, int ctas, int shape, cudaStream_t st) {
    if (g.tiles[0] + g.tiles[1] + g.tiles[2] <= 0) return 0;
    if (shape < 0 || shape >= BATCH_SHAPES || g_resident[shape] <= 0) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(d_counter, 0, BATCH_COUNTERS * sizeof(unsigned long long), st);
    if (e) return (int)e;
    /* the groups' kernels have nothing in common: each begins while the last blocks of the one before it run (300 requests
     * 3,609 -> 3,480 us, a server's 48 requests 1,181 -> 1,083 us, the setups' kernels included) */
    auto group = [&](int i, bool open_pass) {
        return launch_ow_batch(i == 1, tie, open_pass, i == 1 && g.tiles[0] > 0, d_worlds, d_trees, d_reqs + (i ? g.n[0] : 0), g.n[i], g.tiles[i], d_pool, d_counter + i,
                               d_open ? d_open + (i ? open_cap[0] : 0) : nullptr, d_counter + BATCH_GROUPS + i, open_cap[i], d_out, st);
    };
    int rc = group(0, false);
    if (!rc) rc = group(1, false);
    if (rc) return rc;
    if (g.tiles[BATCH_REST] > 0) {
        const MgBatchReq *rq = d_reqs + g.n[0] + g.n[1];
        const int nreq = g.n[BATCH_REST];
        const long long ntiles = g.tiles[BATCH_REST];
        unsigned long long *cnt = d_counter + BATCH_REST;
        int grid = g_resident[shape];
        if (ctas > 0 && ctas < grid) grid = ctas;
        if ((long long)grid > ntiles) grid = (int)ntiles;
        const size_t sm = sizeof(BatchSmem);
        const bool overlap = g.tiles[0] > 0 || g.tiles[1] > 0;
        {
            ProfScope ps_(K_BATCH, st);
            switch (shape) {
            case 1: launch_on(overlap, k_batch<8, 7>, grid, BNT, sm, st, d_worlds, d_trees, rq, nreq, ntiles, d_pool, cnt, d_out); break;
            case 2: launch_on(overlap, k_batch<8, 6>, grid, BNT, sm, st, d_worlds, d_trees, rq, nreq, ntiles, d_pool, cnt, d_out); break;
            case 3: launch_on(overlap, k_batch<8, 8>, grid, BNT, sm, st, d_worlds, d_trees, rq, nreq, ntiles, d_pool, cnt, d_out); break;
            default: launch_on(overlap, k_batch<8, 9>, grid, BNT, sm, st, d_worlds, d_trees, rq, nreq, ntiles, d_pool, cnt, d_out); break;
            }
        }
        count_launch_external();
        if ((e = cudaGetLastError())) return (int)e;
    }
    rc = group(0, true);
    return rc ? rc : group(1, true);
}

}  // namespace mg
