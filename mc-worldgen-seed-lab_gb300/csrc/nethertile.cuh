/* nethertile.cuh -- Nether cells of a 32 x 32-cell tile from tables of lattice nodes (device).
 *
 * The two noises' octaves (8; inputs of at most 1/16 per quart) see the integer quart grid, so, as in the Overworld tiles' shift
 * noises (owtile.cuh), their splits are functions of a column or a row alone and a tile touches a few nodes of each octave's
 * plane: the tables are 64 splits and 9 or 16 nodes per octave for 1,024 cells.  A cell then has 8 octaves from 4 nodes each (the
 * nodes are kept in registers while a warp's rows stay within them) and 5 leaves, the nearest of which it finds directly.
 * The double branch evaluates in the Overworld tiles' fixed point (MgNoise::tile_eq); a cell whose value may have either of two
 * targets is settled when both give the same biome, the rest are evaluated exactly.  4,096 requests of 64 x 64 cells: the per-cell
 * form, bound by 16 FP64 splits a cell and its 14 permutation bytes an octave, took 1,490 us (26.3) and 2,340 us (26.1); this one
 * 489 and 534. */
#ifndef MG_NETHERTILE_CUH
#define MG_NETHERTILE_CUH
#include "owtile.cuh"

namespace mg {

#define NT_W 32     /* tile width and height in cells */
#define NT_OCT 8    /* octaves (lattices) */
#define NT_LEAVES 8
#define NT_NODES 200 /* NT_OCT x 25; at most 16 an octave are used (nether_nodes: 4 per axis at 1/16 per quart) */
#define NT_ROWS 4   /* rows of a thread evaluated together */

/* a leaf: temperature and humidity bounds, squared distance in the other dimensions (their targets are 0) */
struct NetherLeaf {
    int32_t lo0, hi0, lo1, hi1;
    uint32_t rest;
    int32_t biome;
};
struct NetherTile {
    MgLattice lat[NT_OCT];
    union {
        OtShiftF f[NT_OCT][2 * NT_W]; /* columns, then rows */
        OtShiftD d[NT_OCT][2 * NT_W];
    } sh;
    union {
        float4 f[NT_NODES];
        int4 d[NT_NODES];
    } p;
    union {
        float2 f[NT_NODES];
        int2 d[NT_NODES];
    } q;
    int32_t off[NT_OCT + 1], nx[NT_OCT];
    NetherLeaf leaf[NT_LEAVES]; /* in the tree's order */
    int32_t wide;               /* a leaf beyond the 32-bit distances */
};

__host__ __device__ inline int nether_nodes(double f) { return (int)((NT_W - 1) * f * 1.02) + 3; }
/* the worlds whose Nether requests this form takes */
__host__ __device__ inline bool nether_tile_supported(const MgWorldDesc &W) {
    if (W.dim != MG_NETHER || W.ntables > NT_OCT || W.tree_leaves > NT_LEAVES || W.tree_leaves < 1) return false;
    for (int n = 0; n < 2; n++) {
        const MgNoise &N = W.nether[n];
        if (N.base != (n ? 2 * W.nether[0].nlev : 0) || (!W.fmode && N.tile_eq < 0)) return false;
        for (int k = 0; k < N.nlev; k++)
            if (N.fexp[k] > -4 || N.fexp[k] < -40) return false;
    }
    return W.ntables == 2 * (W.nether[0].nlev + W.nether[1].nlev);
}

/* nearest leaf (its place in e.leaf, the first in the tree's order) of target (t, h), |t|, |h| <= 20,000 */
__device__ __forceinline__ int nether_leaf(const NetherTile &e, int n, int32_t t, int32_t h, bool &tied) {
    uint32_t best = 0xFFFFFFFFu;
    int at = 0;
    tied = false;
#pragma unroll 1
    for (int l = 0; l < n; l++) {
        const NetherLeaf f = e.leaf[l];
        const uint32_t a = (uint32_t)max(max(f.lo0 - t, t - f.hi0), 0), b = (uint32_t)max(max(f.lo1 - h, h - f.hi1), 0);
        const uint32_t d = a * a + b * b + f.rest;
        tied = d < best ? false : tied || d == best;
        at = d < best ? l : at;
        best = min(best, d);
    }
    return at;
}

/* a request's part of the tables, by the whole block (barriers around it) */
__device__ __forceinline__ void nether_stage(const MgWorldDesc &W, const MgLattice *__restrict__ pool, const MgTreeNode *__restrict__ tree,
                                             NetherTile &e) {
    const uint4 *a = reinterpret_cast<const uint4 *>(pool);
    uint4 *b = reinterpret_cast<uint4 *>(e.lat);
    for (int i = threadIdx.x; i < W.ntables * (int)(sizeof(MgLattice) / 16); i += blockDim.x) b[i] = a[i];
    if (threadIdx.x < 32) { /* a leaf per lane */
        const int l = threadIdx.x, nl = W.tree_leaves;
        const MgTreeNode n = tree[W.leaf_off + min(l, nl - 1)];
        uint64_t rest = n.d7;
        for (int k = 2; k < 6; k++) {
            const int64_t d = max(max((int)n.lo[k], (int)n.nhi[k]), 0);
            rest += (uint64_t)(d * d);
        }
        int rank = 0;
        for (int m = 0; m < nl; m++) rank += __shfl_sync(0xFFFFFFFFu, (int)n.first, m) < n.first;
        if (l < nl) e.leaf[rank] = NetherLeaf{n.lo[0], -n.nhi[0], n.lo[1], -n.nhi[1], (uint32_t)rest, n.biome};
        /* with bounds within +-12,767 (the packed trees') each of the two squares is below 2^30.01 */
        const bool wide = __any_sync(0xFFFFFFFFu, rest >= (1ULL << 31)) || !rt_packed(tree);
        if (l == 0) e.wide = wide;
    } else if (threadIdx.x == 32) {
        int at = 0;
        for (int l = 0; l < W.ntables; l++) {
            const MgNoise &N = W.nether[l >= W.nether[1].base];
            const int m = nether_nodes(N.freq[(l - N.base) % N.nlev]);
            e.nx[l] = m;
            e.off[l] = at;
            at += m * m;
        }
        e.off[W.ntables] = at;
    }
}

template <bool FM>
__device__ __noinline__ void nether_tile(const MgWorldDesc &W, NetherTile &e, const MgTreeNode *tree, const MgBatchReq &R, int tx0, int tz0,
                                         uint8_t *out) {
    const int t = threadIdx.x, qx0 = R.qx0 + tx0, qz0 = R.qz0 + tz0, noct = W.ntables;
    const bool far = qx0 <= -OT_COORD_LIM || qz0 <= -OT_COORD_LIM || qx0 >= OT_COORD_LIM || qz0 >= OT_COORD_LIM;
    auto noise = [&](int l) -> const MgNoise & { return W.nether[l >= W.nether[1].base]; };
    /* ---- the splits per column and row, the nodes */
    for (int i = far ? noct * 2 * NT_W : t; i < noct * 2 * NT_W; i += (int)blockDim.x) {
        const int l = i / (2 * NT_W), s = i % (2 * NT_W), zc = s >= NT_W, idx = s % NT_W;
        const MgNoise &N = noise(l);
        const MgLattice &L = e.lat[l];
        const double f = N.freq[(l - N.base) % N.nlev], off = zc ? L.oz : L.ox;
        double c0 = (double)(zc ? qz0 : qx0), c = (double)((zc ? qz0 : qx0) + idx);
        if (l - N.base >= N.nlev) { c = c * MG_SECOND_STACK; c0 = c0 * MG_SECOND_STACK; }
        int cell;
        if (FM) {
            OtShiftF v;
            ot_split_f(c, f, off, cell, v.f);
            v.g = v.f - 1.0f;
            v.u = fade<float>(v.f);
            cell -= ifloor(__fma_rn(c0, f, off));
            v.node = zc ? cell * e.nx[l] : cell + e.off[l];
            e.sh.f[l][s] = v;
        } else {
            OtShiftD v;
            ot_split_d(c, f, off, cell, v.f, v.u);
            cell -= ifloor(__fma_rn(c0, f, off));
            v.edge = zc ? cell * e.nx[l] : cell + e.off[l];
            v.pad = 0;
            e.sh.d[l][s] = v;
        }
    }
    for (int i = far ? e.off[noct] : t; i < e.off[noct]; i += (int)blockDim.x) {
        int l = 0;
        while (i >= e.off[l + 1]) l++;
        const MgNoise &N = noise(l);
        const MgLattice &L = e.lat[l];
        const double f = N.freq[(l - N.base) % N.nlev];
        double X = (double)qx0, Z = (double)qz0;
        if (l - N.base >= N.nlev) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
        const int n = i - e.off[l], k = n / e.nx[l];
        const int ib = ifloor(__fma_rn(X, f, L.ox)) + n - k * e.nx[l], kb = ifloor(__fma_rn(Z, f, L.oz)) + k;
        if (FM) ot_node_f(L, false, ib, kb, e.p.f[i], e.q.f[i]);
        else ot_edge(L, false, ot_fix(L.fyd, L.uyd), ib, kb, e.p.d[i], e.q.d[i]);
    }
    __syncthreads();
    /* ---- the cells: a column and NT_ROWS rows at a time */
    const int col = t % NT_W, nl = W.tree_leaves;
    for (int r0 = t / NT_W * NT_ROWS; r0 < NT_W && tz0 + r0 < R.nz; r0 += (int)blockDim.x / NT_W * NT_ROWS) {
        int32_t ta[2][NT_ROWS], tb[2][NT_ROWS]; /* the targets that the cell may have (float branch: ta) */
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const MgNoise &N = W.nether[n];
            if (FM) {
                float acc[NT_ROWS] = {};
#pragma unroll 1
                for (int j = 0; j < (far ? 0 : 2 * N.nlev); j++) { /* first stack, then second: the legacy sum's order */
                    const int l = N.base + j, nx = e.nx[l];
                    const OtShiftF ax = e.sh.f[l][col];
                    const float amp = N.amp_f[j < N.nlev ? j : j - N.nlev], uy = e.lat[l].z0.f.uy;
#pragma unroll
                    for (int r = 0; r < NT_ROWS; r++) {
                        const OtShiftF az = e.sh.f[l][NT_W + r0 + r];
                        acc[r] += amp * ot_octave_f<false>(e.p.f, e.q.f, ax.node + az.node, nx, ax.f, ax.g, ax.u, az.f, az.g, az.u, uy);
                    }
                }
#pragma unroll
                for (int r = 0; r < NT_ROWS; r++) ta[n][r] = tb[n][r] = quantize(acc[r]);
            } else {
                int64_t acc[NT_ROWS] = {}; /* units of 2^-59 */
#pragma unroll 1
                for (int k = 0; k < (far ? 0 : N.nlev); k++) {
                    int64_t lev[NT_ROWS] = {};
#pragma unroll 1
                    for (int st = 0; st < 2; st++) {
                        const int l = N.base + st * N.nlev + k, nx = e.nx[l];
                        const OtShiftD ax = e.sh.d[l][col];
#pragma unroll
                        for (int r = 0; r < NT_ROWS; r++) {
                            const OtShiftD az = e.sh.d[l][NT_W + r0 + r];
                            lev[r] += ot_octave_d(e.p.d, e.q.d, ax.edge + az.edge, nx, ax.f, ax.u, az.f, az.u);
                        }
                    }
#pragma unroll
                    for (int r = 0; r < NT_ROWS; r++) acc[r] = ot_madw((int32_t)(lev[r] >> 31), N.c30[k], acc[r]);
                }
#pragma unroll
                for (int r = 0; r < NT_ROWS; r++) ot_target((int32_t)(acc[r] >> 30), N.tile_eq, 10000.0f * 0x1.0p-29f, ta[n][r], tb[n][r]);
            }
        }
#pragma unroll
        for (int r = 0; r < NT_ROWS; r++) {
            const int row = r0 + r;
            if (tx0 + col >= R.nx || tz0 + row >= R.nz) continue;
            bool ok = !far && !e.wide && max(max(abs(ta[0][r]), abs(tb[0][r])), max(abs(ta[1][r]), abs(tb[1][r]))) <= 20000;
            int b = 0;
            if (ok) {
                bool tied;
                b = e.leaf[nether_leaf(e, nl, ta[0][r], ta[1][r], tied)].biome;
                ok = !(tied && R.tie == MG_TIE_CHUNK_CELL); /* a tied cell's candidate chain */
                if (!FM) {
                    const int d0 = tb[0][r] - ta[0][r], d1 = tb[1][r] - ta[1][r];
                    if (d0 | d1) { /* one target of two: both; else open */
                        ok &= (unsigned)d0 + (unsigned)d1 <= 1u;
                        ok &= e.leaf[nether_leaf(e, nl, tb[0][r], tb[1][r], tied)].biome == b;
                        ok &= !(tied && R.tie == MG_TIE_CHUNK_CELL);
                    }
                }
            }
            if (!ok) {
                const int qx = qx0 + col, qz = qz0 + row;
                if (R.tie == MG_TIE_CHUNK_CELL) {
                    b = cell_chunk<FM, MG_NETHER>(W, W.spline, e.lat, tree, qx, R.qy, qz);
                } else {
                    int32_t tg[6];
                    cell_target<FM, MG_NETHER>(W, W.spline, e.lat, qx, R.qy, qz, tg);
                    uint64_t d;
                    b = tree[tree_search(tree, tg, -1, d)].biome;
                }
            }
            put_id(out + R.out_off + (size_t)(tz0 + row) * R.nx + tx0 + col, b);
        }
    }
    __syncthreads(); /* the tables are free for the next tile */
}

}  // namespace mg
#endif
