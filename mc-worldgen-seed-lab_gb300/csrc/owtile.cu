/* owtile.cu -- the Overworld over areas: the batched form's requests, quart grids and the drop-in block map, by persistent
 * kernels over 16 x 16-cell tiles whose octaves read tables of lattice nodes (owtile.cuh). */
#include <cuda_runtime.h>
#include <stdint.h>

#include "batch.h"
#include "batchdev.cuh"
#include "launch.h"
#include "overlap.cuh"
#include "owtile.cuh"
#include "prof.h"
#include "warpcell.cuh"

namespace mg {

/* nodes a tile's table holds: the shift noises' (about 610) or the climate octaves' (about 680 on average) */
#define OT_CAP_F 1024

/* a tile of a request; kept in shared memory so that its fields are read where they are used (held in registers over the
 * whole tile they made the double branch's kernel spill: 72.1 -> 68.7 ms) */
struct OtTile {
    MgBatchReq r;
    int req, tile;
};
struct OtSmemF {
    MgLattice lat[MG_MAX_TABLES];
    float4 np[OT_CAP_F];
    float2 nq[OT_CAP_F];
    OtShiftF sh[2 * OT_MAXLEV][4 * OT_TABW]; /* per lattice: X + ox, X + oy, Z + oz, Z + ox (a column or row each) */
    OtOctF oct[MG_MAX_TABLES];            /* the climate octaves in evaluation order */
    OtBuild build, sbuild;                /* climate and shift tables */
    int lo[2], hi[2];                     /* range of the shifted x and z over the tile, in 1/16 of a quart from its corner */
    int state, over;
    OtTile cur[2]; /* this tile and the next */
    uint16_t hint[OT_NT]; /* each thread's last leaf: where its next R-tree search starts */
};

/* the per-cell form, for a tile whose nodes do not fit or beyond the tables' coordinates (out of line: rare) */
template <bool FM>
static __device__ __noinline__ void ot_cell_plain(const MgWorldDesc &W, const MgLattice *T, int qx, int qy, int qz, int32_t *tg) {
    int32_t t[6];
    climate_ow<FM>(W, W.spline, T, qx, qy, qz, t);
    for (int k = 0; k < 6; k++) tg[k] = t[k];
}

/* a search's leaf as the next search's hint (a leaf found by the lane alone is a node of the tree: no hint) */
__device__ __forceinline__ uint16_t ot_hint(const MgWorldDesc &W, int leaf) {
    return (uint16_t)(leaf >= W.leaf_off ? leaf - W.leaf_off : 0);
}
/* where tiles come from: a batch's requests through its work queue, or one grid's tiles in turn (reqs null) */
struct OtWork {
    const MgWorldDesc *worlds;
    const MgTreeNode *const *trees; /* per world; or, for one grid, null and `tree` */
    const MgTreeNode *tree;
    const MgBatchReq *reqs;
    int nreq;
    long long ntiles;
    const MgLattice *pool;
    unsigned long long *counter;
    MgOpenCell *open; /* cells left to the exact evaluation, their counter and the room for them */
    unsigned long long *nopen;
    long long open_cap;
    uint8_t *out;
    MgBatchReq one;             /* one grid */
    int64_t zseed;              /* OT_BLOCK: zoom seed, first block, spacing, block y */
    int32_t x0, z0, step, y;
    const int32_t *xyz;         /* or the blocks themselves (k_ow_sparse) */
    ChainRec *rec;              /* OT_CHAIN */
};
/* next tile and its request (one whole warp calls it); prev: the CTA's last tile of one grid, -1 at first */
__device__ __forceinline__ void ot_next(OtTile &n, const OtWork &K, int prev) {
    if (!K.reqs) {
        if ((threadIdx.x & 31) == 0) {
            const long long tile = prev < 0 ? (long long)blockIdx.x : (long long)prev + gridDim.x;
            n.r = K.one;
            n.req = tile < K.ntiles ? 0 : -1;
            n.tile = (int)tile;
        }
        return;
    }
    long long tile = 0;
    if ((threadIdx.x & 31) == 0) tile = (long long)atomicAdd(K.counter, 1ULL);
    tile = __shfl_sync(0xFFFFFFFFu, tile, 0);
    const int r = tile < K.ntiles ? find_req(K.reqs, K.nreq, tile) : -1;
    if ((threadIdx.x & 31) == 0) {
        n.req = r;
        if (r >= 0) {
            n.r = K.reqs[r];
            n.tile = (int)(tile - n.r.tile0);
        }
    }
}
/* the quart cell of tile cell (tx, tz) of the grid, counted from (qx0, qz0) and quart y0 */
template <int MODE>
__device__ __forceinline__ void ot_cell(const OtWork &K, int tx, int tz, int qx0, int qz0, int qy0, int &dx, int &dz, int &dy) {
    int cx, cy, cz;
    zoom_cell(K.zseed, K.x0 + tx * K.step, K.y, K.z0 + tz * K.step, cx, cy, cz);
    dx = cx - qx0;
    dz = cz - qz0;
    dy = cy - qy0;
}
__device__ __forceinline__ int ot_clamp_y(const MgWorldDesc &W, int qy) {
    const int lo = W.min_y >> 2, hi = lo + (W.height >> 2) - 1;
    return qy < lo ? lo : (qy > hi ? hi : qy);
}
/* one cell by the per-lane exact forms: a cell left open that has no room in the record, or one of many recorded ones */
template <bool FM, int MODE>
__device__ __noinline__ void ot_exact(const OtWork &K, const MgWorldDesc &W, const MgLattice *T, const MgTreeNode *tree, int qx, int qy,
                                      int qz, long long o) {
    if (MODE == OT_CHUNK || MODE == OT_BLOCK) {
        put_id(K.out + o, cell_chunk<FM, MG_OVERWORLD>(W, W.spline, T, tree, qx, qy, qz));
        return;
    }
    int32_t tg[6];
    climate_ow<FM>(W, W.spline, T, qx, qy, qz, tg);
    uint64_t d;
    if (MODE == OT_CHAIN) {
        bool tied;
        const int leaf = tree_search_tie(tree, tg, d, tied);
        ChainRec &r = K.rec[o];
        for (int k = 0; k < 6; k++) r.tg[k] = tg[k];
        r.d = d;
        r.leaf = leaf;
        r.tie = tied;
        put_id(K.out + o, tree[leaf].biome);
    } else {
        put_id(K.out + o, tree[tree_search_scattered(tree, tg, -1, d)].biome);
    }
}
/* leave a cell open: recorded, or evaluated here when the record is full */
template <bool FM, int MODE>
__device__ __forceinline__ void ot_leave_open(const OtWork &K, const MgWorldDesc &W, const MgLattice *T, const MgTreeNode *tree, int req,
                                              int cell, int qx, int qy, int qz, long long o) {
    const unsigned long long k = K.open_cap > 0 ? atomicAdd(K.nopen, 1ULL) : ~0ULL;
    if (k < (unsigned long long)K.open_cap) K.open[k] = MgOpenCell{req, cell};
    else ot_exact<FM, MODE>(K, W, T, tree, qx, qy, qz, o);
}

/* Float branch (26.3 on), bit for bit the per-cell form's operations.  Bound by instruction issue (69 % of peak; the octaves'
 * separately rounded lerps, the splits' mantissa shifts, the tree scan).  64 registers and 55 KB of shared memory: 4 CTAs,
 * 32 warps per SM.  The uneven batch's 70.8 M float-branch cells: 47.6 ms in the per-cell form, 34.2 ms here (8 of it the tree). */
template <int MODE>
__global__ void __launch_bounds__(OT_NT, 4) k_ow_f(const __grid_constant__ OtWork K) {
    extern __shared__ uint4 smem_raw[];
    OtSmemF &sm = *reinterpret_cast<OtSmemF *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int col = ot_col(), row = ot_row();
    if (t == 0) sm.state = -1;
    sm.hint[t] = 0;
    overlap_next();
    if (warp == 0) ot_next(sm.cur[0], K, -1);
    __syncthreads();
    for (int c = 0;; c ^= 1) {
        if (sm.cur[c].req < 0) break;
        const int tile = sm.cur[c].tile;
        const MgBatchReq &R = sm.cur[c].r;
        const MgWorldDesc &W = K.worlds[R.world];
        const MgNoise &O = W.noise[0];
        const int nlev = O.nlev, nsh = 2 * nlev, nclim = W.ntables - nsh;
        const int tw = mg_parts(R.nx, OT_W);
        const int tx0 = (tile % tw) * OT_W, tz0 = (tile / tw) * OT_W;
        /* first quart cell of the tile (of a block map: the lowest the zoom can give) */
        const int qx0 = MODE == OT_BLOCK ? (K.x0 + tx0 * K.step - 2) >> 2 : R.qx0 + tx0;
        const int qz0 = MODE == OT_BLOCK ? (K.z0 + tz0 * K.step - 2) >> 2 : R.qz0 + tz0;
        const int qy0 = MODE == OT_BLOCK ? (K.y - 2) >> 2 : R.qy;
        /* beyond the world border the wrap may move a cell: the per-cell form takes the tile */
        const bool far = qx0 <= -OT_COORD_LIM || qz0 <= -OT_COORD_LIM || qx0 >= OT_COORD_LIM || qz0 >= OT_COORD_LIM;
        if (R.state != sm.state) { /* the request's lattices, octave constants and shift table layout */
            const uint4 *a = reinterpret_cast<const uint4 *>(K.pool + R.state);
            uint4 *b = reinterpret_cast<uint4 *>(sm.lat);
            for (int i = t; i < W.ntables * (int)(sizeof(MgLattice) / 16); i += OT_NT) b[i] = a[i];
            __syncthreads();
            if (t == 0) sm.state = R.state;
            sm.hint[t] = 0; /* another request's world may have fewer leaves */
            if (t < nclim) { /* octave t in evaluation order */
                int n = 1;
                while (n < MG_OW_NOISES - 1 && t + nsh >= W.noise[n + 1].base) n++;
                const MgNoise &N = W.noise[n];
                const int e = t + nsh - N.base, k = e >> 1;
                const int l = N.base + (e & 1) * N.nlev + k;
                const MgLattice &L = sm.lat[l];
                sm.build.nx[t] = (int16_t)l; /* the climate tables' lattice (their row length is the range's) */
                OtOctF &o = sm.oct[t];
                o.ox = L.ox;
                o.oz = L.oz;
                o.f = N.freq[k];
                o.amp = N.amp_f[k];
                o.uy = L.z0.f.uy;
            }
            if (warp == 7) { /* shift tables: lattice j's (x, 0, z) form is table 2 j, its (x, y, 0) form 2 j + 1 */
                const int m = lane < 2 * nsh ? ot_shift_nodes(O.freq[(lane >> 1) % nlev]) : 0;
                int off = (m * m + 31) / 32, n = off;
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, off, d);
                    if (lane >= d) off += v;
                }
                sm.sbuild.unit0[lane] = lane < 2 * nsh ? off - n : 0x7FFFFFFF;
                sm.sbuild.unit0[lane + 32] = 0x7FFFFFFF;
                sm.sbuild.n[lane] = (int16_t)(m * m);
                sm.sbuild.nx[lane] = (int16_t)m;
                sm.sbuild.inv[lane] = (m ? (65536 + m - 1) / m : 0);
                if (lane == 31) sm.sbuild.units = off;
            }
            __syncthreads();
        }
        /* ---- 1: the shift noises' splits per column and row, and their nodes */
        for (int e = far ? nsh * 4 * OT_TABW : t; e < nsh * 4 * OT_TABW; e += OT_NT) {
            const int j = e / (4 * OT_TABW), q = e % (4 * OT_TABW), fam = q / OT_TABW, idx = q % OT_TABW;
            const MgLattice &L = sm.lat[j];
            const double f = O.freq[j % nlev];
            const double off = fam == 0 || fam == 3 ? L.ox : (fam == 1 ? L.oy : L.oz);
            double c = fam < 2 ? (double)(qx0 + idx) : (double)(qz0 + idx), c0 = fam < 2 ? (double)qx0 : (double)qz0;
            if (j >= nlev) { c = c * MG_SECOND_STACK; c0 = c0 * MG_SECOND_STACK; }
            OtShiftF s;
            int i;
            ot_split_f(c, f, off, i, s.f);
            s.g = s.f - 1.0f;
            s.u = fade<float>(s.f);
            const int tab = 2 * j + (fam & 1), rel = i - ifloor(__fma_rn(c0, f, off));
            /* x-like coordinates (families 0 and 3) step one node, the others a row; the table's place with the first */
            s.node = fam == 0 || fam == 3 ? rel + 32 * sm.sbuild.unit0[tab] : rel * sm.sbuild.nx[tab];
            sm.sh[j][q] = s;
        }
        for (int u = far ? sm.sbuild.units : warp; u < sm.sbuild.units; u += OT_NT / 32) {
            const int tab = ot_find_unit(sm.sbuild, u);
            const int n = (u - sm.sbuild.unit0[tab]) * 32 + lane;
            if (n >= sm.sbuild.n[tab]) continue;
            const int j = tab >> 1, z0 = tab & 1, nx = sm.sbuild.nx[tab];
            const int k = n * sm.sbuild.inv[tab] >> 16, i = n - k * nx;
            const MgLattice &L = sm.lat[j];
            const double f = O.freq[j % nlev];
            double X = (double)qx0, Z = (double)qz0;
            if (j >= nlev) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
            const int ib = ifloor(__fma_rn(z0 ? Z : X, f, L.ox)), kb = ifloor(__fma_rn(z0 ? X : Z, f, z0 ? L.oy : L.oz));
            const int at = 32 * sm.sbuild.unit0[tab] + n;
            ot_node_f(L, z0, ib + i, kb + k, sm.np[at], sm.nq[at]);
        }
        if (t == 0) {
            sm.lo[0] = sm.lo[1] = 0x7FFFFFFF;
            sm.hi[0] = sm.hi[1] = -0x7FFFFFFF;
            sm.over = far;
        }
        __syncthreads();
        /* ---- 2: the shift noises and the shifted coordinates of the cell */
        const bool in = tx0 + col < R.nx && tz0 + row < R.nz;
        int dx = col, dz = row, dy = 0; /* the cell, from the tile's first */
        if (MODE == OT_BLOCK) {
            if (in) ot_cell<MODE>(K, tx0 + col, tz0 + row, qx0, qz0, qy0, dx, dz, dy);
            else dx = dz = 0;
        }
        double x = 0.0, z = 0.0;
        if (!far) {
            float sa = 0.0f, sb = 0.0f;
#pragma unroll 1
            for (int q = 0; q < nsh; q++) { /* level by level, first stack then second: each sum in its order */
                const int k = q >> 1, j = (q & 1) * nlev + k;
                const OtShiftF ax = sm.sh[j][dx], by = sm.sh[j][OT_TABW + dx], az = sm.sh[j][2 * OT_TABW + dz],
                               bx = sm.sh[j][3 * OT_TABW + dz];
                const float amp = O.amp_f[k];
                sa += amp * ot_octave_f<false>(sm.np, sm.nq, ax.node + az.node, sm.sbuild.nx[2 * j], ax.f, ax.g, ax.u, az.f,
                                               az.g, az.u, sm.lat[j].z0.f.uy);
                sb += amp * ot_octave_f<true>(sm.np, sm.nq, bx.node + by.node, sm.sbuild.nx[2 * j + 1], bx.f, bx.g, bx.u, by.f,
                                              by.g, by.u, sm.lat[j].z0.f.uz);
            }
            const float sx = sa * 4.0f, sz = sb * 4.0f;
            x = (double)(qx0 + dx) + (double)sx;
            z = (double)(qz0 + dz) + (double)sz;
            const int rx = __float2int_rd(((float)dx + sx) * 16.0f), rz = __float2int_rd(((float)dz + sz) * 16.0f);
            const int x0 = __reduce_min_sync(0xFFFFFFFFu, in ? rx : 0x7FFFFFFF), x1 = __reduce_max_sync(0xFFFFFFFFu, in ? rx : -0x7FFFFFFF);
            const int z0 = __reduce_min_sync(0xFFFFFFFFu, in ? rz : 0x7FFFFFFF), z1 = __reduce_max_sync(0xFFFFFFFFu, in ? rz : -0x7FFFFFFF);
            if (lane == 0 && x0 <= x1) {
                atomicMin(&sm.lo[0], x0);
                atomicMax(&sm.hi[0], x1);
                atomicMin(&sm.lo[1], z0);
                atomicMax(&sm.hi[1], z1);
            }
        }
        __syncthreads();
        /* ---- 3: the climate octaves' node ranges (warp 0), the next tile (warp 1) */
        if (warp == 0 && !far) {
            /* one sixteenth more on either side covers the float sum's rounding */
            const double xl = (double)qx0 + (double)(sm.lo[0] - 1) * 0.0625, xh = (double)qx0 + (double)(sm.hi[0] + 2) * 0.0625;
            const double zl = (double)qz0 + (double)(sm.lo[1] - 1) * 0.0625, zh = (double)qz0 + (double)(sm.hi[1] + 2) * 0.0625;
            int nodes = 0, units = 0, bad = 0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int e = lane + 32 * h;
                OtRange g{0, 0, 0, 0};
                int n = 0;
                if (e < nclim) {
                    OtOctF &o = sm.oct[e];
                    const double c = (e & 1) ? MG_SECOND_STACK : 1.0; /* every noise starts at an even octave */
                    g.ib = ifloor(__fma_rn(xl * c, o.f, o.ox));
                    g.kb = ifloor(__fma_rn(zl * c, o.f, o.oz));
                    const int nx = ifloor(__fma_rn(xh * c, o.f, o.ox)) - g.ib + 2, nz = ifloor(__fma_rn(zh * c, o.f, o.oz)) - g.kb + 2;
                    bad |= nx > 32 || nz > 32;
                    g.nx = nx;
                    n = nx * nz;
                }
                int a = n, b = (n + 31) / 32;
                for (int d = 1; d < 32; d <<= 1) {
                    const int va = __shfl_up_sync(0xFFFFFFFFu, a, d), vb = __shfl_up_sync(0xFFFFFFFFu, b, d);
                    if (lane >= d) { a += va; b += vb; }
                }
                g.off = nodes + a - n;
                if (e < nclim) sm.oct[e].r = g;
                sm.build.unit0[e] = e < nclim ? units + b - (n + 31) / 32 : 0x7FFFFFFF;
                sm.build.n[e] = (int16_t)n;
                sm.build.inv[e] = (g.nx ? (65536 + g.nx - 1) / g.nx : 0);
                nodes += __shfl_sync(0xFFFFFFFFu, a, 31);
                units += __shfl_sync(0xFFFFFFFFu, b, 31);
            }
            if (__any_sync(0xFFFFFFFFu, bad) || nodes > OT_CAP_F) {
                if (lane == 0) sm.over = 1;
            } else if (lane == 0) {
                sm.build.units = units;
            }
        } else if (warp == 1) {
            ot_next(sm.cur[c ^ 1], K, tile);
        }
        __syncthreads();
        const bool over = sm.over != 0;
        /* ---- 4: the climate octaves' nodes */
        if (!over) {
            for (int u = warp; u < sm.build.units; u += OT_NT / 32) {
                const int e = ot_find_unit(sm.build, u);
                const int n = (u - sm.build.unit0[e]) * 32 + lane;
                if (n >= sm.build.n[e]) continue;
                const OtRange g = sm.oct[e].r;
                const int k = n * sm.build.inv[e] >> 16, i = n - k * g.nx;
                ot_node_f(sm.lat[sm.build.nx[e]], false, g.ib + i, g.kb + k, sm.np[g.off + n], sm.nq[g.off + n]);
            }
        }
        __syncthreads();
        /* ---- 5: the climate noises, the targets, the R-tree */
        int32_t tg[6] = {0, 0, 0, 0, 0, 0};
        if (in) {
            if (!over) {
                double xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
                /* kept in registers: the compiler would form the products again in every octave (FP64 pipe) */
                asm volatile("" : "+d"(xc), "+d"(zc));
                float v[MG_OW_NOISES - 1];
                int e = 0;
#pragma unroll 1
                for (int n = 0; n < MG_OW_NOISES - 1; n++) { /* one copy of the octave's code for the five noises */
                    const int end = e + 2 * W.noise[n + 1].nlev;
                    float acc = 0.0f;
#pragma unroll 1
                    for (; e < end; e++) {
                        const OtOctF o = sm.oct[e];
                        int ia, ib;
                        float fa, fb;
                        ot_split_f((e & 1) ? xc : x, o.f, o.ox, ia, fa);
                        ot_split_f((e & 1) ? zc : z, o.f, o.oz, ib, fb);
                        const int at = o.r.off + (ib - o.r.kb) * o.r.nx + (ia - o.r.ib);
                        acc += o.amp * ot_octave_f<false>(sm.np, sm.nq, at, o.r.nx, fa, fa - 1.0f, fade<float>(fa), fb, fb - 1.0f,
                                                          fade<float>(fb), o.uy);
                    }
#pragma unroll
                    for (int k = 0; k < MG_OW_NOISES - 1; k++) v[k] = n == k ? acc : v[k];
                }
                climate_finish_f(W, W.spline, v[0], v[1], v[2], v[3], v[4],
                                 (MODE == OT_CHUNK || MODE == OT_BLOCK ? ot_clamp_y(W, qy0 + dy) : qy0) * 4, tg);
            } else {
                ot_cell_plain<true>(W, sm.lat, qx0 + dx, MODE == OT_CHUNK || MODE == OT_BLOCK ? ot_clamp_y(W, qy0 + dy) : qy0, qz0 + dz, tg);
            }
        }
        const MgTreeNode *tree = K.trees ? K.trees[R.world] : K.tree;
        uint64_t d = 0;
        bool tied = false;
        int leaf;
        if (MODE == OT_ENGINE) leaf = tree_search_warp(tree, W, tg, in, sm.hint[t]);
        else leaf = tree_search_tie_warp(tree, W, tg, in, d, tied, sm.hint[t]);
        if (in) {
            sm.hint[t] = ot_hint(W, leaf);
            const int cell = (int)((unsigned)(tile / tw * OT_W + row) * (unsigned)R.nx) + tile % tw * OT_W + col; /* of a cell in the request: fits */
            const int64_t o = R.out_off + cell;
            if (MODE == OT_CHAIN) {
                ChainRec &q = K.rec[o];
                for (int k = 0; k < 6; k++) q.tg[k] = tg[k];
                q.d = d;
                q.leaf = leaf;
                q.tie = tied;
            }
            /* a tied cell's candidate chain is left to the launch that follows */
            if ((MODE == OT_CHUNK || MODE == OT_BLOCK) && tied)
                ot_leave_open<true, MODE>(K, W, sm.lat, tree, sm.cur[c].req, cell, qx0 + dx, qy0 + dy, qz0 + dz, o);
            else put_id(K.out + o, tree[leaf].biome);
        }
        __syncthreads(); /* the tables are free for the next tile */
    }
    overlap_wait();
}

/* ============================================================================ double branch */
#define OT_CAP_D 896 /* edges a tile's table holds */

struct OtSmemD {
    MgLattice lat[MG_MAX_TABLES];
    int4 ep[OT_CAP_D];
    int2 eq[OT_CAP_D];
    OtShiftD sh[2 * OT_MAXLEV][4 * OT_TABW];
    OtOctD oct[MG_MAX_TABLES];
    int64_t oct_o[MG_MAX_TABLES][2]; /* the climate octaves' offsets in units of 2^-32 */
    int2 oct_b[MG_MAX_TABLES];       /* their first cells */
    OtFix fix[MG_MAX_TABLES], sfix[OT_SHIFT_TABS]; /* climate octaves; shift tables */
    OtBuild build, sbuild;
    int lo[2], hi[2];
    int state, over;
    OtTile cur[2]; /* this tile and the next */
    uint16_t hint[OT_NT];
    int32_t depth[2]; /* depth gradient and offset constant at quart y0 and y0 + 1, units of 2^-28 */
};

/* Double branch (26.1, 26.2).  The per-cell form was bound by the FP64 pipe (12 exact shift octaves, 348 operations of 446 a
 * cell at two lanes per SM and clock) beside 40 octaves of 64 x 64-bit products; here nothing per cell uses FP64 and an octave
 * is 11 32 x 32-bit products.  Bound by instruction issue and the wide multiplies.  The uneven batch's 151.6 M double-branch
 * cells: 222.5 ms in the per-cell form, 66.1 ms here (22 of it the tree), and 0.5 ms in k_ow_open. */
template <int MODE>
__global__ void __launch_bounds__(OT_NT, 4) k_ow_d(const __grid_constant__ OtWork K) {
    extern __shared__ uint4 smem_raw[];
    OtSmemD &sm = *reinterpret_cast<OtSmemD *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int col = ot_col(), row = ot_row();
    if (t == 0) sm.state = -1;
    sm.hint[t] = 0;
    overlap_next();
    if (warp == 0) ot_next(sm.cur[0], K, -1);
    __syncthreads();
    for (int c = 0;; c ^= 1) {
        if (sm.cur[c].req < 0) break;
        const int tile = sm.cur[c].tile;
        const MgBatchReq &R = sm.cur[c].r;
        const MgWorldDesc &W = K.worlds[R.world];
        const MgNoise &O = W.noise[0];
        const int nlev = O.nlev, nsh = 2 * nlev, nclim = W.ntables - nsh;
        const int tw = mg_parts(R.nx, OT_W);
        const int tx0 = (tile % tw) * OT_W, tz0 = (tile / tw) * OT_W;
        /* first quart cell of the tile (of a block map: the lowest the zoom can give) */
        const int qx0 = MODE == OT_BLOCK ? (K.x0 + tx0 * K.step - 2) >> 2 : R.qx0 + tx0;
        const int qz0 = MODE == OT_BLOCK ? (K.z0 + tz0 * K.step - 2) >> 2 : R.qz0 + tz0;
        const int qy0 = MODE == OT_BLOCK ? (K.y - 2) >> 2 : R.qy;
        const bool far = qx0 <= -OT_COORD_LIM || qz0 <= -OT_COORD_LIM || qx0 >= OT_COORD_LIM || qz0 >= OT_COORD_LIM;
        if (R.state != sm.state) { /* the request's lattices, octave constants and shift table layout */
            const uint4 *a = reinterpret_cast<const uint4 *>(K.pool + R.state);
            uint4 *b = reinterpret_cast<uint4 *>(sm.lat);
            for (int i = t; i < W.ntables * (int)(sizeof(MgLattice) / 16); i += OT_NT) b[i] = a[i];
            __syncthreads();
            if (t == 0) sm.state = R.state;
            sm.hint[t] = 0; /* another request's world may have fewer leaves */
            if (t < nclim) { /* octave t in evaluation order */
                int n = 1;
                while (n < MG_OW_NOISES - 1 && t + nsh >= W.noise[n + 1].base) n++;
                const MgNoise &N = W.noise[n];
                const int e = t + nsh - N.base, k = e >> 1;
                const int l = N.base + (e & 1) * N.nlev + k;
                const MgLattice &L = sm.lat[l];
                sm.build.nx[t] = (int16_t)l; /* the climate tables' lattice */
                sm.oct_o[t][0] = __double2ll_rn(L.ox * 0x1.0p32);
                sm.oct_o[t][1] = __double2ll_rn(L.oz * 0x1.0p32);
                sm.oct[t].k = -N.fexp[k];
                sm.oct[t].c30 = N.c30[k];
                sm.fix[t] = ot_fix(L.fyd, L.uyd);
            } else if (t >= 64 && t < 64 + 2 * nsh) { /* shift tables: lattice j's (x, 0, z) form is 2 j, its (x, y, 0) form 2 j + 1 */
                const MgLattice &L = sm.lat[(t - 64) >> 1];
                sm.sfix[t - 64] = (t & 1) ? ot_fix(L.fzd, L.uzd) : ot_fix(L.fyd, L.uyd);
            }
            if (warp == 7) {
                const int m = lane < 2 * nsh ? ot_shift_nodes(O.freq[(lane >> 1) % nlev]) : 0;
                int off = (m * m + 31) / 32, n = off;
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, off, d);
                    if (lane >= d) off += v;
                }
                sm.sbuild.unit0[lane] = lane < 2 * nsh ? off - n : 0x7FFFFFFF;
                sm.sbuild.unit0[lane + 32] = 0x7FFFFFFF;
                sm.sbuild.n[lane] = (int16_t)(m * m);
                sm.sbuild.nx[lane] = (int16_t)m;
                sm.sbuild.inv[lane] = (m ? (65536 + m - 1) / m : 0);
                if (lane == 31) sm.sbuild.units = off;
            }
            __syncthreads();
        }
        /* ---- 1: the shift noises' splits per column and row, and their edges */
        for (int e = far ? nsh * 4 * OT_TABW : t; e < nsh * 4 * OT_TABW; e += OT_NT) {
            const int j = e / (4 * OT_TABW), q = e % (4 * OT_TABW), fam = q / OT_TABW, idx = q % OT_TABW;
            const MgLattice &L = sm.lat[j];
            const double f = O.freq[j % nlev];
            const double off = fam == 0 || fam == 3 ? L.ox : (fam == 1 ? L.oy : L.oz);
            double c = fam < 2 ? (double)(qx0 + idx) : (double)(qz0 + idx), c0 = fam < 2 ? (double)qx0 : (double)qz0;
            if (j >= nlev) { c = c * MG_SECOND_STACK; c0 = c0 * MG_SECOND_STACK; }
            int i;
            OtShiftD s;
            ot_split_d(c, f, off, i, s.f, s.u);
            const int tab = 2 * j + (fam & 1), rel = i - ifloor(__fma_rn(c0, f, off));
            s.edge = fam == 0 || fam == 3 ? rel + 32 * sm.sbuild.unit0[tab] : rel * sm.sbuild.nx[tab];
            s.pad = 0;
            sm.sh[j][q] = s;
        }
        for (int u = far ? sm.sbuild.units : warp; u < sm.sbuild.units; u += OT_NT / 32) {
            const int tab = ot_find_unit(sm.sbuild, u);
            const int n = (u - sm.sbuild.unit0[tab]) * 32 + lane;
            if (n >= sm.sbuild.n[tab]) continue;
            const int j = tab >> 1, z0 = tab & 1, nx = sm.sbuild.nx[tab];
            const int k = n * sm.sbuild.inv[tab] >> 16, i = n - k * nx;
            const MgLattice &L = sm.lat[j];
            const double f = O.freq[j % nlev];
            double X = (double)qx0, Z = (double)qz0;
            if (j >= nlev) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
            const int ib = ifloor(__fma_rn(z0 ? Z : X, f, L.ox)), kb = ifloor(__fma_rn(z0 ? X : Z, f, z0 ? L.oy : L.oz));
            const int at = 32 * sm.sbuild.unit0[tab] + n;
            ot_edge(L, z0, sm.sfix[tab], ib + i, kb + k, sm.ep[at], sm.eq[at]);
        }
        if (t == 0) {
            sm.lo[0] = sm.lo[1] = 0x7FFFFFFF;
            sm.hi[0] = sm.hi[1] = -0x7FFFFFFF;
            sm.over = far;
        } else if (t >= OT_NT - 2) { /* a block map's cells lie at two heights */
            const int i = OT_NT - 1 - t, qy = MODE == OT_CHUNK || MODE == OT_BLOCK ? ot_clamp_y(W, qy0 + i) : qy0;
            sm.depth[i] = (int32_t)__double2ll_rn((depth_grad_d(W, qy * 4) + W.off_d) * 0x1.0p28);
        }
        __syncthreads();
        /* ---- 2: the shift noises and the shifted coordinates of the cell (units of 2^-32) */
        const bool in = tx0 + col < R.nx && tz0 + row < R.nz;
        int dx = col, dz = row, dy = 0; /* the cell, from the tile's first */
        if (MODE == OT_BLOCK) {
            if (in) ot_cell<MODE>(K, tx0 + col, tz0 + row, qx0, qz0, qy0, dx, dz, dy);
            else dx = dz = 0;
        }
        int64_t x = 0, z = 0;
        if (!far) {
            int64_t sa = 0, sb = 0; /* units of 2^-59 */
#pragma unroll 1
            for (int k = 0; k < nlev; k++) {
                int64_t va = 0, vb = 0;
#pragma unroll
                for (int st = 0; st < 2; st++) {
                    const int j = st * nlev + k;
                    const OtShiftD ax = sm.sh[j][dx], by = sm.sh[j][OT_TABW + dx], az = sm.sh[j][2 * OT_TABW + dz],
                                   bx = sm.sh[j][3 * OT_TABW + dz];
                    va += ot_octave_d(sm.ep, sm.eq, ax.edge + az.edge, sm.sbuild.nx[2 * j], ax.f, ax.u, az.f, az.u);
                    vb += ot_octave_d(sm.ep, sm.eq, bx.edge + by.edge, sm.sbuild.nx[2 * j + 1], bx.f, bx.u, by.f, by.u);
                }
                const int32_t c = O.c30[k];
                sa = ot_madw((int32_t)(va >> 31), c, sa);
                sb = ot_madw((int32_t)(vb >> 31), c, sb);
            }
            x = ((int64_t)(qx0 + dx) << 32) + (sa >> 25); /* the noise times 4 */
            z = ((int64_t)(qz0 + dz) << 32) + (sb >> 25);
            const int rx = dx * 16 + (int)(sa >> 53), rz = dz * 16 + (int)(sb >> 53);
            const int x0 = __reduce_min_sync(0xFFFFFFFFu, in ? rx : 0x7FFFFFFF), x1 = __reduce_max_sync(0xFFFFFFFFu, in ? rx : -0x7FFFFFFF);
            const int z0 = __reduce_min_sync(0xFFFFFFFFu, in ? rz : 0x7FFFFFFF), z1 = __reduce_max_sync(0xFFFFFFFFu, in ? rz : -0x7FFFFFFF);
            if (lane == 0 && x0 <= x1) {
                atomicMin(&sm.lo[0], x0);
                atomicMax(&sm.hi[0], x1);
                atomicMin(&sm.lo[1], z0);
                atomicMax(&sm.hi[1], z1);
            }
        }
        __syncthreads();
        /* ---- 3: the climate octaves' edge ranges (warp 0), the next tile (warp 1) */
        if (warp == 0 && !far) {
            const int64_t xl = ((int64_t)qx0 << 32) + ((int64_t)sm.lo[0] << 28), xh = ((int64_t)qx0 << 32) + ((int64_t)(sm.hi[0] + 1) << 28);
            const int64_t zl = ((int64_t)qz0 << 32) + ((int64_t)sm.lo[1] << 28), zh = ((int64_t)qz0 << 32) + ((int64_t)(sm.hi[1] + 1) << 28);
            const int64_t cxl = xl + __mul64hi(xl, OT_STACK_C), cxh = xh + __mul64hi(xh, OT_STACK_C);
            const int64_t czl = zl + __mul64hi(zl, OT_STACK_C), czh = zh + __mul64hi(zh, OT_STACK_C);
            int edges = 0, units = 0, bad = 0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int e = lane + 32 * h;
                int n = 0, nx = 0, ib = 0, kb = 0;
                if (e < nclim) {
                    const int k = sm.oct[e].k;
                    const int64_t ox = sm.oct_o[e][0], oz = sm.oct_o[e][1];
                    ib = ot_hi((((e & 1) ? cxl : xl) >> k) + ox);
                    kb = ot_hi((((e & 1) ? czl : zl) >> k) + oz);
                    nx = ot_hi((((e & 1) ? cxh : xh) >> k) + ox) - ib + 1;
                    const int nz = ot_hi((((e & 1) ? czh : zh) >> k) + oz) - kb + 2;
                    bad |= nx > 31 || nz > 32;
                    n = nx * nz;
                }
                int a = n, b = (n + 31) / 32;
                for (int d = 1; d < 32; d <<= 1) {
                    const int va = __shfl_up_sync(0xFFFFFFFFu, a, d), vb = __shfl_up_sync(0xFFFFFFFFu, b, d);
                    if (lane >= d) { a += va; b += vb; }
                }
                if (e < nclim) {
                    OtOctD &o = sm.oct[e];
                    o.ox = sm.oct_o[e][0] - ((int64_t)ib << 32);
                    o.oz = sm.oct_o[e][1] - ((int64_t)kb << 32);
                    o.nx = nx;
                    o.off = edges + a - n;
                    sm.oct_b[e] = make_int2(ib, kb);
                }
                sm.build.unit0[e] = e < nclim ? units + b - (n + 31) / 32 : 0x7FFFFFFF;
                sm.build.n[e] = (int16_t)n;
                sm.build.inv[e] = (nx ? (65536 + nx - 1) / nx : 0);
                edges += __shfl_sync(0xFFFFFFFFu, a, 31);
                units += __shfl_sync(0xFFFFFFFFu, b, 31);
            }
            if (__any_sync(0xFFFFFFFFu, bad) || edges > OT_CAP_D) {
                if (lane == 0) sm.over = 1;
            } else if (lane == 0) {
                sm.build.units = units;
            }
        } else if (warp == 1) {
            ot_next(sm.cur[c ^ 1], K, tile);
        }
        __syncthreads();
        const bool over = sm.over != 0;
        /* ---- 4: the climate octaves' edges */
        if (!over) {
            for (int u = warp; u < sm.build.units; u += OT_NT / 32) {
                const int e = ot_find_unit(sm.build, u);
                const int n = (u - sm.build.unit0[e]) * 32 + lane;
                if (n >= sm.build.n[e]) continue;
                const int nx = sm.oct[e].nx, off = sm.oct[e].off;
                const int k = n * sm.build.inv[e] >> 16, i = n - k * nx;
                const int2 b = sm.oct_b[e];
                ot_edge(sm.lat[sm.build.nx[e]], false, sm.fix[e], b.x + i, b.y + k, sm.ep[off + n], sm.eq[off + n]);
            }
        }
        __syncthreads();
        /* ---- 5: the climate noises, the targets, the R-tree */
        bool ok = in && !over;
        int32_t ta[6] = {0, 0, 0, 0, 0, 0}, tb[6] = {0, 0, 0, 0, 0, 0}; /* the targets the cell may have: [ta, tb] */
        if (ok) {
            const int64_t xc = x + __mul64hi(x, OT_STACK_C), zc = z + __mul64hi(z, OT_STACK_C);
            int32_t v[MG_OW_NOISES - 1]; /* units of 2^-29 */
            int e = 0;
#pragma unroll 1
            for (int n = 0; n < MG_OW_NOISES - 1; n++) { /* one copy of the octave's code for the five noises */
                const int end = e + 2 * W.noise[n + 1].nlev;
                int64_t acc = 0; /* units of 2^-59 */
#pragma unroll 1
                for (; e < end; e += 2) {
                    int64_t lev = 0;
                    int32_t c = 0;
#pragma unroll
                    for (int st = 0; st < 2; st++) {
                        const OtOctD o = sm.oct[e + st];
                        const int64_t sx = ((st ? xc : x) >> o.k) + o.ox, sz = ((st ? zc : z) >> o.k) + o.oz;
                        const int at = o.off + ot_hi(sz) * o.nx + ot_hi(sx);
                        lev += ot_octave_d(sm.ep, sm.eq, at, o.nx, (int32_t)((uint32_t)sx >> 1), ot_fade31((uint32_t)sx),
                                           (int32_t)((uint32_t)sz >> 1), ot_fade31((uint32_t)sz));
                        c = o.c30;
                    }
                    acc = ot_madw((int32_t)(lev >> 31), c, acc);
                }
#pragma unroll
                for (int k = 0; k < MG_OW_NOISES - 1; k++) v[k] = n == k ? (int32_t)(acc >> 30) : v[k];
            }
            const bool out17 = max(max(abs(qx0), abs(qz0)) + OT_W, 0) >= 1 << 17;
            int32_t eq[MG_OW_NOISES];
#pragma unroll
            for (int n = 1; n < MG_OW_NOISES; n++) eq[n] = out17 ? W.noise[n].tile_eq_far : W.noise[n].tile_eq;
            float es;
            ot_climate_targets(W, W.spline, v, eq, sm.depth[MODE == OT_BLOCK ? dy : 0], ta, tb, es);
            ok = es < 1.0f;
        }
        /* at most one target open, between two neighbouring values: both are looked up, and the cell is settled when they
         * give the same biome (nearly always: a step is 1e-4 of the range) */
        int amb = 0;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            amb += tb[k] - ta[k];
            ok &= (unsigned)(tb[k] - ta[k]) <= 1u;
        }
        ok &= amb <= 1;
        const MgTreeNode *tree = K.trees ? K.trees[R.world] : K.tree;
        const int cell = (int)((unsigned)(tile / tw * OT_W + row) * (unsigned)R.nx) + tile % tw * OT_W + col; /* of a cell in the request: fits */
        const int64_t o = R.out_off + cell;
        int biome = -1; /* (OT_CHAIN: the leaf) */
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) { /* the lower targets, then the upper ones of cells with two */
            const bool act = ok && (pass == 0 || amb);
            if (pass && !__any_sync(0xFFFFFFFFu, act)) break;
            int32_t t6[6];
#pragma unroll
            for (int k = 0; k < 6; k++) t6[k] = pass ? tb[k] : ta[k];
            uint64_t d = 0;
            bool tied = false;
            int leaf;
            bool sure = pass == 0 && amb;
            if (MODE == OT_ENGINE) leaf = tree_search_warp<true>(tree, W, t6, act, sm.hint[t], &sure);
            else leaf = tree_search_tie_warp<true>(tree, W, t6, act, d, tied, sm.hint[t], &sure);
            if (sure) amb = 0; /* the upper target's leaf is the same */
            if (act) {
                sm.hint[t] = ot_hint(W, leaf);
                if (MODE == OT_CHAIN) {
                    ChainRec &q = K.rec[o];
                    for (int k = 0; k < 6; k++) q.tg[k] = t6[k];
                    q.d = d;
                    q.leaf = leaf;
                    q.tie = tied;
                }
                const int b = MODE == OT_CHAIN ? leaf : tree[leaf].biome;
                ok = pass == 0 || b == biome;
                /* a tied cell's chain needs the target (OT_CHAIN: a record's target is read only for tied cells) */
                if (MODE == OT_CHUNK || MODE == OT_BLOCK) ok &= !tied;
                if (MODE == OT_CHAIN) ok &= !(tied && amb);
                biome = b;
            }
        }
        if (in) {
            if (ok) put_id(K.out + o, MODE == OT_CHAIN ? tree[biome].biome : biome);
            else ot_leave_open<false, MODE>(K, W, sm.lat, tree, sm.cur[c].req, cell, qx0 + dx, qy0 + dy, qz0 + dz, o);
        }
        __syncthreads(); /* the tables are free for the next tile */
    }
    overlap_wait();
}

/* ============================================================================ sparse block maps, long point lists
 * Blocks more than 4 apart or anywhere: neighbouring cells share too few nodes for a tile's tables, so each is evaluated by its
 * lane: the float branch by the per-cell form, the double branch in the tiles' fixed point with its octaves' edges built on the way
 * (ot_cell_d; per cell in double, its shift noises took 864 FP64 operations), beyond the tables' coordinates by the per-cell form
 * too.  Tied cells and open targets are left to k_ow_open like the tiles'.  The lattices, spline and fixed coordinates' parts are in
 * shared memory; warps take 8 x 4 cells, whose tree search they share up to 16 blocks apart (a box of 4 x 8 chunks of terrain) and
 * do one by one beyond and for points.  256 x 256 blocks, spacing 16: 26.1 531 -> 205 us, 26.3 379 -> 237 us; spacing 37: 578 ->
 * 313, 552 -> 229 (its search shared: 324 and 288). */
struct OtSparse {
    WcStage st;
    OtFix fix[MG_MAX_TABLES], fz[2 * OT_MAXLEV]; /* of the y plane; the shift's z plane */
    int64_t off[MG_MAX_TABLES][2];               /* offsets in units of 2^-32 */
    int32_t depth[2];
};
template <bool FM>
__global__ void __launch_bounds__(128, 4) k_ow_sparse(const __grid_constant__ OtWork K) {
    extern __shared__ uint4 smem_raw[];
    OtSparse &sm = *reinterpret_cast<OtSparse *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const MgWorldDesc &W = K.worlds[0];
    const MgSpline &S = sm.st.spline;
    const MgTreeNode *tree = K.tree;
    const int nx = K.one.nx, nz = K.one.nz, tw = mg_parts(nx, 16), qy0 = (K.y - 2) >> 2;
    wc_stage(sm.st, W, K.pool, t, 128);
    overlap_next();
    __syncthreads();
    if (!FM) {
        ot_cell_fix(W, sm.st.lat, sm.fix, sm.fz, sm.off, t, 128);
        if (t >= 126) sm.depth[127 - t] = (int32_t)__double2ll_rn((depth_grad_d(W, ot_clamp_y(W, qy0 + 127 - t) * 4) + W.off_d) * 0x1.0p28);
        __syncthreads();
    }
    for (long long tile = blockIdx.x; tile < K.ntiles; tile += gridDim.x) {
        const int ix = K.xyz ? (int)tile * 128 + t : (int)(tile % tw) * 16 + (warp & 1) * 8 + (lane & 7);
        const int iz = K.xyz ? 0 : (int)(tile / tw) * 8 + (warp >> 1) * 4 + (lane >> 3);
        const bool in = ix < nx && iz < nz;
        int cx = 0, cy = qy0, cz = 0;
        if (in) {
            const int32_t *p = K.xyz + 3 * (size_t)ix;
            if (K.xyz) zoom_cell(K.zseed, p[0], p[1], p[2], cx, cy, cz);
            else zoom_cell(K.zseed, K.x0 + ix * K.step, K.y, K.z0 + iz * K.step, cx, cy, cz);
        }
        bool ok = in;
        int32_t ta[6] = {0, 0, 0, 0, 0, 0}, amb = 0;
        if (FM) {
            if (in) climate_ow<true>(W, S, sm.st.lat, cx, ot_clamp_y(W, cy), cz, ta);
        } else {
            ok = in && cx > -OT_COORD_LIM && cx < OT_COORD_LIM && cz > -OT_COORD_LIM && cz < OT_COORD_LIM;
            if (ok) {
                int32_t v[MG_OW_NOISES - 1], tb[6], eq[MG_OW_NOISES];
                ot_cell_d(W, sm.st.lat, sm.fix, sm.fz, sm.off, cx, cz, v, eq);
                float es;
                const int32_t depth = K.xyz ? (int32_t)__double2ll_rn((depth_grad_d(W, ot_clamp_y(W, cy) * 4) + W.off_d) * 0x1.0p28)
                                            : sm.depth[cy - qy0];
                ot_climate_targets(W, S, v, eq, depth, ta, tb, es);
                ok = es < 1.0f;
#pragma unroll
                for (int k = 0; k < 6; k++) {
                    amb += tb[k] - ta[k];
                    ok &= (unsigned)(tb[k] - ta[k]) <= 1u;
                }
                ok &= amb <= 1;
            } else if (in && (long long)nx * nz > OT_FEW_BLOCKS) {
                ot_cell_plain<false>(W, sm.st.lat, cx, ot_clamp_y(W, cy), cz, ta);
                ok = true;
            }
        }
        uint64_t d;
        bool tied = false, sure = amb != 0;
        int leaf;
        if (!K.xyz && K.step <= 16) {
            if (FM) leaf = tree_search_tie_warp(tree, W, ta, ok, d, tied);
            else leaf = tree_search_tie_warp<true>(tree, W, ta, ok, d, tied, -1, &sure);
        } else {
            leaf = tree_search_lanes(tree, W, ta, ok, &tied);
            sure = false;
        }
        if (!in) continue;
        const int cell = iz * nx + ix;
        if (ok && !tied && (!amb || sure)) put_id(K.out + cell, tree[leaf].biome);
        else ot_leave_open<FM, OT_BLOCK>(K, W, sm.st.lat, tree, 0, cell, cx, cy, cz, cell);
    }
}

/* the open cells: up to 65,536 by a warp each (25 us for the first, then its throughput), more by a thread each (200 us for any
 * number).  One grid's lattices and spline are copied to shared memory by each block; a batch's are read through L1.  24 warps
 * per SM: a cell by a warp is a chain of latencies, so its rate is the warps in flight.  Under the chunk-cell rule a block takes
 * each cell: its tied chain's cells at once (wc_block_chunk). */
#define OT_OPEN_NT 128
#define OT_OPEN_SMEM sizeof(WcStage)
template <bool FM, int MODE>
__global__ void __launch_bounds__(OT_OPEN_NT, 6) k_ow_open(const __grid_constant__ OtWork K) {
    extern __shared__ uint4 smem_raw[];
    WcStage &s = *reinterpret_cast<WcStage *>(smem_raw);
    if (!K.reqs) wc_stage(s, K.worlds[0], K.pool, threadIdx.x, OT_OPEN_NT); /* while the tiles' last blocks run */
    overlap_wait(); /* the cells are recorded */
    const long long n = min((long long)*K.nopen, K.open_cap);
    const bool by_warp = n <= 65536 || MODE == OT_CHUNK || MODE == OT_BLOCK;
    const int lane = threadIdx.x & 31;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x, threads = (long long)gridDim.x * blockDim.x;
    if (!by_warp) {
        for (long long i = id; i < n; i += threads) {
            const MgOpenCell c = K.open[i];
            const MgBatchReq R = K.reqs ? K.reqs[c.req] : K.one;
            const int iz = c.cell / R.nx, ix = c.cell - iz * R.nx;
            ot_exact<FM, MODE>(K, K.worlds[R.world], K.pool + R.state, K.trees ? K.trees[R.world] : K.tree, R.qx0 + ix, R.qy, R.qz0 + iz,
                               R.out_off + c.cell);
        }
        return;
    }
    if ((long long)blockIdx.x * (MODE == OT_CHUNK || MODE == OT_BLOCK ? 1 : OT_OPEN_NT / 32) >= n) return;
    __syncthreads();
    __shared__ WcStep steps[MODE == OT_CHUNK || MODE == OT_BLOCK ? WC_STEPS : 1];
    constexpr bool chains = MODE == OT_CHUNK || MODE == OT_BLOCK; /* a block per cell, else a warp */
    for (long long i = chains ? (long long)blockIdx.x : id >> 5; i < n; i += chains ? (long long)gridDim.x : threads >> 5) {
        const MgOpenCell c = K.open[i];
        const MgBatchReq R = K.reqs ? K.reqs[c.req] : K.one;
        const MgWorldDesc &W = K.worlds[R.world];
        const MgTreeNode *tree = K.trees ? K.trees[R.world] : K.tree;
        const MgLattice *T = K.reqs ? K.pool + R.state : s.lat;
        const MgSpline &S = K.reqs ? W.spline : s.spline;
        const int iz = c.cell / R.nx, ix = c.cell - iz * R.nx;
        int qx = R.qx0 + ix, qy = R.qy, qz = R.qz0 + iz;
        const long long o = R.out_off + c.cell;
        if (MODE == OT_BLOCK) {
            const int32_t *p = K.xyz + 3 * (size_t)c.cell;
            if (K.xyz) wc_zoom(K.zseed, p[0], p[1], p[2], qx, qy, qz);
            else wc_zoom(K.zseed, K.x0 + ix * K.step, K.y, K.z0 + iz * K.step, qx, qy, qz);
        }
        if (chains) {
            const int b = wc_block_chunk<FM, MG_OVERWORLD, OT_OPEN_NT / 32>(W, S, T, tree, qx, qy, qz, steps);
            if (threadIdx.x == 0) put_id(K.out + o, b);
            __syncthreads();
            continue;
        }
        int32_t tg[6];
        wc_target<FM, MG_OVERWORLD>(W, S, T, qx, qy, qz, tg);
        uint64_t d;
        bool tied;
        const int leaf = wc_search(tree, W, tg, d, tied);
        if (lane) continue;
        if (MODE == OT_CHAIN) {
            ChainRec &r = K.rec[o];
            for (int k = 0; k < 6; k++) r.tg[k] = tg[k];
            r.d = d;
            r.leaf = leaf;
            r.tie = tied;
        }
        put_id(K.out + o, tree[leaf].biome);
    }
}

/* ---------------------------------------------------------------- host side */
/* a world whose Overworld requests the tile kernels take: power-of-two frequencies of at most 1/2 per quart (the wrap is
 * the identity up to the world border, and the tables' sizes hold), shift levels and nodes within the tables */
bool ow_tile_supported(const MgWorldDesc &W) {
    if (W.dim != MG_OVERWORLD) return false;
    if (!W.fmode) { /* the fixed point's ranges */
        for (int n = 0; n < MG_OW_NOISES; n++)
            if (W.noise[n].tile_eq < 0) return false;
        if (W.rf_eq < 0 || !W.rf_tile) return false;
        if (!(fmax(fabs(W.grad_from_d), fabs(W.grad_to_d)) + fabs(W.off_d) < OT_DEPTH_LIM) || W.grad_from_y == W.grad_to_y) return false;
    }
    if (W.noise[0].base != 0 || W.noise[0].nlev > OT_MAXLEV) return false;
    int base = 0, cap = 0;
    for (int n = 0; n < MG_OW_NOISES; n++) {
        const MgNoise &N = W.noise[n];
        if (N.base != base || N.nlev < 1) return false;
        base += 2 * N.nlev;
        for (int k = 0; k < N.nlev; k++)
            if (N.fexp[k] > -1 || N.fexp[k] < -40) return false;
    }
    if (base != W.ntables || base - 2 * W.noise[0].nlev > 64 || base > MG_MAX_TABLES) return false;
    for (int k = 0; k < W.noise[0].nlev; k++) {
        const int m = ot_shift_nodes(W.noise[0].freq[k]);
        cap += 4 * ((m * m + 31) / 32) * 32;
    }
    return cap <= (W.fmode ? OT_CAP_F : OT_CAP_D);
}
/* In the double branch the tiles leave every cell beyond the tables' coordinates open.  Up to `few` k_ow_open has sooner, by a warp
 * (a block under the chunk-cell rule) each, than a thread each (FP64: two lanes per SM and clock): 26.1 beyond 2^23 quarts, grids of
 * 16 x 16 cells 40 against 161 us, 64 x 64 81 against 165, maps of 16 x 16 blocks 72 against 183, of 64 x 64 275 against 187.  More
 * would fill the record and be done one by one, so an area of more cells that reaches there takes the forms with a thread per cell
 * (a grid of 256 x 256 cells 450 us in the tiles, 272 so), and a batch's requests that do all of them. */
bool ow_beyond(bool fm, long long few, long long qx0, long long qz0, long long qx1, long long qz1, long long cells) {
    const long long lim = OT_COORD_LIM - 2 * OT_W;
    return !fm && cells > few && (qx0 <= -lim || qz0 <= -lim || qx1 >= lim || qz1 >= lim);
}
long long ow_tiles(int nx, int nz) { return (long long)mg_parts(nx, OT_W) * mg_parts(nz, OT_W); }

static int g_ow_resident[2][4]; /* CTAs per SM x SMs by branch and mode (ow_prepare; callers hold the ABI lock) */
template <int MODE>
static int prepare_mode(int sms) {
    int rc = (int)cudaFuncSetAttribute(k_ow_d<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OtSmemD)), n = 0;
    if (!rc) rc = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ow_d<MODE>, OT_NT, sizeof(OtSmemD));
    g_ow_resident[0][MODE] = (n > 0 ? n : 1) * sms;
    if (!rc) rc = (int)cudaFuncSetAttribute(k_ow_f<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OtSmemF));
    if (!rc) rc = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ow_f<MODE>, OT_NT, sizeof(OtSmemF));
    g_ow_resident[1][MODE] = (n > 0 ? n : 1) * sms;
    return rc;
}
int ow_prepare() {
    static int prepared_dev = -1; /* the attributes are per device and set once */
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    if (prepared_dev == dev) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int rc = prepare_mode<OT_ENGINE>(sms);
    if (!rc) rc = prepare_mode<OT_CHUNK>(sms);
    if (!rc) rc = prepare_mode<OT_BLOCK>(sms);
    if (!rc) rc = prepare_mode<OT_CHAIN>(sms);
    if (!rc) prepared_dev = dev;
    return rc;
}
long long ow_open_cap(long long cells) { return cells > 0 ? cells / 32 + 4096 : 0; }

template <int MODE>
static void tiles_t(bool fm, bool overlap, const OtWork &K, int grid, cudaStream_t st) {
    if (fm) launch_on(overlap, k_ow_f<MODE>, grid, OT_NT, sizeof(OtSmemF), st, K);
    else launch_on(overlap, k_ow_d<MODE>, grid, OT_NT, sizeof(OtSmemD), st, K);
}
static int launch_tiles(bool fm, int mode, bool overlap, const OtWork &K, cudaStream_t st) {
    const int resident = g_ow_resident[fm][mode];
    if (resident <= 0) return (int)cudaErrorInvalidValue;
    const int grid = (long long)resident < K.ntiles ? resident : (int)K.ntiles;
    {
        ProfScope ps_(fm ? K_OW_TILE_F : K_OW_TILE_D, st);
        switch (mode) {
        case OT_CHUNK: tiles_t<OT_CHUNK>(fm, overlap, K, grid, st); break;
        case OT_BLOCK: tiles_t<OT_BLOCK>(fm, overlap, K, grid, st); break;
        case OT_CHAIN: tiles_t<OT_CHAIN>(fm, overlap, K, grid, st); break;
        default: tiles_t<OT_ENGINE>(fm, overlap, K, grid, st); break;
        }
    }
    count_launch_external();
    return (int)cudaGetLastError();
}
template <int MODE>
static void open_t(bool fm, const OtWork &K, int grid, cudaStream_t st) {
    if (fm) launch_on(true, k_ow_open<true, MODE>, grid, OT_OPEN_NT, OT_OPEN_SMEM, st, K);
    else launch_on(true, k_ow_open<false, MODE>, grid, OT_OPEN_NT, OT_OPEN_SMEM, st, K);
}
static int launch_open(bool fm, int mode, const OtWork &K, cudaStream_t st) {
    if (!K.open || K.open_cap <= 0) return 0;
    const int grid = 6 * 152;
    {
        ProfScope ps_(K_OW_OPEN, st);
        switch (mode) {
        case OT_CHUNK: open_t<OT_CHUNK>(fm, K, grid, st); break;
        case OT_BLOCK: open_t<OT_BLOCK>(fm, K, grid, st); break;
        case OT_CHAIN: if (!fm) launch_on(true, k_ow_open<false, OT_CHAIN>, grid, OT_OPEN_NT, OT_OPEN_SMEM, st, K); break;
        default: if (!fm) launch_on(true, k_ow_open<false, OT_ENGINE>, grid, OT_OPEN_NT, OT_OPEN_SMEM, st, K); break;
        }
    }
    count_launch_external();
    return (int)cudaGetLastError();
}

int launch_ow_batch(bool fm, int tie, bool open_pass, bool overlap, const MgWorldDesc *d_worlds, const MgTreeNode *const *d_trees,
                    const MgBatchReq *d_reqs, int nreq, long long ntiles, const MgLattice *d_pool, unsigned long long *d_counter,
                    MgOpenCell *d_open, unsigned long long *d_nopen, long long open_cap, uint8_t *d_out, cudaStream_t st) {
    if (ntiles <= 0) return 0;
    OtWork K{};
    K.worlds = d_worlds;
    K.trees = d_trees;
    K.reqs = d_reqs;
    K.nreq = nreq;
    K.ntiles = ntiles;
    K.pool = d_pool;
    K.counter = d_counter;
    K.open = d_open;
    K.nopen = d_nopen;
    K.open_cap = d_open ? open_cap : 0;
    K.out = d_out;
    const int mode = tie == MG_TIE_CHUNK_CELL ? OT_CHUNK : OT_ENGINE;
    return open_pass ? (fm && mode == OT_ENGINE ? 0 : launch_open(fm, mode, K, st)) : launch_tiles(fm, mode, overlap, K, st);
}

/* ---- one grid: scratch for the open cells' record (a counter, then the cells) */
static long long grid_open_cap(bool fm, int mode, long long cells) {
    return fm && (mode == OT_ENGINE || mode == OT_CHAIN) ? 0 : ow_open_cap(cells);
}
size_t ow_grid_scratch_bytes(const MgWorldDesc &W, bool chunk_rule, long long cells) {
    const long long cap = grid_open_cap(W.fmode != 0, chunk_rule ? OT_BLOCK : OT_CHAIN, cells);
    return cap > 0 ? 16 + (size_t)cap * sizeof(MgOpenCell) : 0;
}
static int open_scratch(bool fm, int mode, OtWork &K, void *scratch, cudaStream_t st) {
    K.open_cap = scratch ? grid_open_cap(fm, mode, (long long)K.one.nx * K.one.nz) : 0;
    if (K.open_cap <= 0) return 0;
    K.nopen = (unsigned long long *)scratch;
    K.open = (MgOpenCell *)((uint8_t *)scratch + 16);
    return (int)cudaMemsetAsync(K.nopen, 0, sizeof(unsigned long long), st);
}
static int grid_run(const MgWorldDesc &W, int mode, OtWork &K, void *scratch, cudaStream_t st) {
    const bool fm = W.fmode != 0;
    K.ntiles = ow_tiles(K.one.nx, K.one.nz);
    int rc = ow_prepare();
    if (!rc) rc = open_scratch(fm, mode, K, scratch, st);
    if (rc) return rc;
    rc = launch_tiles(fm, mode, false, K, st);
    return rc ? rc : launch_open(fm, mode, K, st);
}
int launch_ow_quart_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int qx0,
                         int qz0, int nx, int nz, int qy, ChainRec *rec, uint8_t *out, void *scratch, cudaStream_t st) {
    OtWork K{};
    K.worlds = d_world;
    K.tree = tree;
    K.pool = state;
    K.out = out;
    K.rec = rec;
    K.one.qx0 = qx0;
    K.one.qz0 = qz0;
    K.one.nx = nx;
    K.one.nz = nz;
    K.one.qy = qy;
    return grid_run(W, rec ? OT_CHAIN : OT_ENGINE, K, scratch, st);
}
/* blocks more than 4 apart, points, double-branch maps beyond the tables' coordinates */
static int sparse_run(const MgWorldDesc &W, OtWork &K, void *scratch, cudaStream_t st) {
    const bool fm = W.fmode != 0;
    K.ntiles = K.xyz ? mg_parts(K.one.nx, 128) : (long long)mg_parts(K.one.nx, 16) * mg_parts(K.one.nz, 8);
    int rc = open_scratch(fm, OT_BLOCK, K, scratch, st);
    if (rc) return rc;
    rc = (int)(fm ? cudaFuncSetAttribute(k_ow_sparse<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OtSparse))
                  : cudaFuncSetAttribute(k_ow_sparse<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OtSparse)));
    if (rc) return rc;
    const unsigned grid = (unsigned)(K.ntiles < 4 * 152 ? K.ntiles : 4 * 152);
    {
        ProfScope ps_(K_BLOCKGRID, st);
        if (fm) k_ow_sparse<true><<<grid, 128, sizeof(OtSparse), st>>>(K);
        else k_ow_sparse<false><<<grid, 128, sizeof(OtSparse), st>>>(K);
    }
    count_launch_external();
    rc = (int)cudaGetLastError();
    return rc ? rc : launch_open(fm, OT_BLOCK, K, st);
}
bool ow_block_grid_supported(const MgWorldDesc &W, int x0, int z0) {
    return ow_tile_supported(W) && x0 >= INT32_MIN + 16 && z0 >= INT32_MIN + 16;
}
int launch_ow_block_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int64_t zseed,
                         int x0, int z0, int nx, int nz, int step, int y, const int32_t *xyz, uint8_t *out, void *scratch,
                         cudaStream_t st) {
    OtWork K{};
    K.worlds = d_world;
    K.tree = tree;
    K.pool = state;
    K.out = out;
    K.one.nx = nx;
    K.one.nz = nz;
    K.zseed = zseed;
    K.x0 = x0;
    K.z0 = z0;
    K.step = step;
    K.y = y;
    K.xyz = xyz;
    const bool far = ow_beyond(W.fmode != 0, OT_FEW_BLOCKS, x0 >> 2, z0 >> 2, (x0 + (long long)(nx - 1) * step) >> 2,
                               (z0 + (long long)(nz - 1) * step) >> 2, (long long)nx * nz);
    return !xyz && step <= 4 && !far ? grid_run(W, OT_BLOCK, K, scratch, st) : sparse_run(W, K, scratch, st);
}

}  // namespace mg
