/* warpcell.cuh -- one cell per warp: the exact climate of a cell with one octave per lane, the R-tree search with one leaf
 * per lane, BiomeManager's zoom with one candidate per lane, and the chunk-cell rule on top (device).
 *
 * The per-lane forms (climate.cuh) run a cell's 52 octaves and its tree search in series: right where a warp's lanes are all
 * busy with cells of their own, but a lone cell (a point query, a tied cell's candidate chain) then takes 52 octaves' and some
 * 150 node visits' latency while 31 lanes wait.  Here every lane evaluates at most 3 octaves; the values are the per-lane
 * forms' (oct_f, oct_d), summed in their order.  A lone cell's time is its chains of dependent loads (permutation bytes, spline
 * points, tree nodes), so the seed's lattices and the spline are copied to shared memory first, 24 KB in parallel. */
#ifndef MG_WARPCELL_CUH
#define MG_WARPCELL_CUH
#include "climate.cuh"

namespace mg {

#define WC_FULL 0xFFFFFFFFu

/* a seed's lattices and its world's spline in shared memory */
struct WcStage {
    MgLattice lat[MG_MAX_TABLES];
    MgSpline spline;
};
/* copied by threads t of nt (a barrier among them must follow) */
__device__ __forceinline__ void wc_stage(WcStage &s, const MgWorldDesc &W, const MgLattice *__restrict__ src, int t, int nt) {
    const uint4 *a = reinterpret_cast<const uint4 *>(src);
    uint4 *b = reinterpret_cast<uint4 *>(s.lat);
#pragma unroll 4
    for (int i = t; i < W.ntables * (int)(sizeof(MgLattice) / 16); i += nt) b[i] = a[i];
    if (W.dim != MG_OVERWORLD) return;
    const uint4 *c = reinterpret_cast<const uint4 *>(&W.spline);
    uint4 *d = reinterpret_cast<uint4 *>(&s.spline);
#pragma unroll 4
    for (int i = t; i < (int)(sizeof(MgSpline) / 16); i += nt) d[i] = c[i];
}

/* octave e of a noise-major list (a noise's levels, first then second stack of each) starting at noise n0: its noise, level
 * and stack */
__device__ __forceinline__ void wc_octave(const MgNoise *N, int n0, int nn, int e, int &n, int &k, int &st) {
    n = n0;
    while (n < nn - 1 && e >= 2 * N[n].nlev) {
        e -= 2 * N[n].nlev;
        n++;
    }
    k = e >> 1;
    st = e & 1;
}
/* the term of octave e at (a, 0, b) (z0: (a, b, 0)), second stack's inputs ac, bc: float branch amp * octave, double branch
 * amp * octave * value factor, as the sums take it */
template <bool FM>
__device__ __forceinline__ double wc_term(const MgNoise &N, const MgLattice *__restrict__ T, int k, int st, double a, double b,
                                          double ac, double bc, bool z0) {
    const MgLattice *L = T + N.base + st * N.nlev + k;
    if (FM) return (double)(N.amp_f[k] * oct_f(L, st ? ac : a, st ? bc : b, N.freq[k], N.fexp[k], z0));
    return N.amp_d[k] * oct_d(L, st ? ac : a, st ? bc : b, N.freq[k], N.fexp[k], z0) * N.vf_d[k];
}
/* value of the noise whose terms start at octave e0 of the lanes' lists (t0: octaves 0-31, t1: 32-63), for the lane's own e0
 * and level count (lanes with nlev 0 get 0): the float branch adds level by level, first stack then second; legacy stack by
 * stack; the double branch each stack, then the two.  All lanes call it with the same `most` >= every lane's nlev. */
template <bool FM>
__device__ __forceinline__ double wc_sum(double t0, double t1, int e0, int nlev, int most, bool legacy, double vfac) {
    float f = 0.0f;
    double s0 = 0.0, s1 = 0.0;
    for (int i = 0; i < 2 * most; i++) {
        const int e = FM && legacy ? e0 + (i < nlev ? 2 * i : 2 * (i - nlev) + 1) : e0 + i;
        const double u0 = __shfl_sync(WC_FULL, t0, e & 31), u1 = __shfl_sync(WC_FULL, t1, e & 31);
        const double u = e < 32 ? u0 : u1;
        if (i < 2 * nlev) {
            if (FM) f += (float)u;
            else if (i & 1) s1 += u;
            else s0 += u;
        }
    }
    return FM ? (double)f : (s0 + s1) * vfac;
}
/* six quantised targets of quart cell (qx, qy, qz), the same in every lane (all 32 call it) */
template <bool FM, int DIM>
__device__ __noinline__ void wc_target(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T, int qx, int qy, int qz,
                                       int32_t *tg) {
    const int lane = threadIdx.x & 31;
    const double X = (double)qx, Z = (double)qz, Xc = X * MG_SECOND_STACK, Zc = Z * MG_SECOND_STACK;
    int n, k, st;
    if (DIM == MG_NETHER) {
        const int na = 2 * W.nether[0].nlev, tot = na + 2 * W.nether[1].nlev;
        double t0 = 0.0;
        if (lane < tot) {
            wc_octave(W.nether, 0, 2, lane, n, k, st);
            t0 = wc_term<FM>(W.nether[n], T, k, st, X, Z, Xc, Zc, false);
        }
        const int m = lane & 1;
        const double v = wc_sum<FM>(t0, 0.0, m ? na : 0, W.nether[m].nlev, max(W.nether[0].nlev, W.nether[1].nlev), true, W.nether[m].vfac);
        const float t = (float)__shfl_sync(WC_FULL, v, 0), h = (float)__shfl_sync(WC_FULL, v, 1);
        tg[0] = quantize(t);
        tg[1] = quantize(h);
        tg[2] = tg[3] = tg[4] = tg[5] = 0;
        return;
    }
    const MgNoise &O = W.noise[0];
    const int nsh = 2 * O.nlev, nclim = W.ntables - nsh;
    /* shift: lanes 0 .. nsh - 1 ShiftA (x, 0, z), the next nsh ShiftB (z, x, 0) */
    double t = 0.0;
    if (lane < 2 * nsh) {
        const bool b = lane >= nsh;
        wc_octave(W.noise, 0, 1, b ? lane - nsh : lane, n, k, st);
        t = wc_term<FM>(O, T, k, st, b ? Z : X, b ? X : Z, b ? Zc : Xc, b ? Xc : Zc, b);
    }
    const double sh = wc_sum<FM>(t, 0.0, lane & 1 ? nsh : 0, O.nlev, O.nlev, false, O.vfac);
    const double sa = __shfl_sync(WC_FULL, sh, 0), sb = __shfl_sync(WC_FULL, sh, 1);
    double x, z;
    if (FM) {
        x = X + (double)((float)sa * 4.0f);
        z = Z + (double)((float)sb * 4.0f);
    } else {
        x = X + sa * 4.0;
        z = Z + sb * 4.0;
    }
    const double xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
    double t0 = 0.0, t1 = 0.0;
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        if (lane + 32 * r >= nclim) continue;
        wc_octave(W.noise, 1, MG_OW_NOISES, lane + 32 * r, n, k, st);
        const double v = wc_term<FM>(W.noise[n], T, k, st, x, z, xc, zc, false);
        if (r) t1 = v;
        else t0 = v;
    }
    __syncwarp();
    /* lane j < 5 sums noise j + 1 */
    int e0 = 0, most = 0;
    const int mine = min(lane, MG_OW_NOISES - 2) + 1;
    for (int q = 1; q < MG_OW_NOISES; q++) {
        if (q < mine) e0 += 2 * W.noise[q].nlev;
        most = max(most, W.noise[q].nlev);
    }
    const double v = wc_sum<FM>(t0, t1, e0, W.noise[mine].nlev, most, false, W.noise[mine].vfac);
    double nv[MG_OW_NOISES - 1];
#pragma unroll
    for (int q = 0; q < MG_OW_NOISES - 1; q++) nv[q] = __shfl_sync(WC_FULL, v, q);
    if (FM) climate_finish_f(W, S, (float)nv[0], (float)nv[1], (float)nv[2], (float)nv[3], (float)nv[4], qy * 4, tg);
    else climate_finish_d(W, S, nv[0], nv[1], nv[2], nv[3], nv[4], qy * 4, tg);
}

/* tree_search_tie for one target, the same in every lane: the lanes take a cluster's groups and a group's leaves, one each.
 * The nearest leaf (node index), its distance, whether a second leaf has it. */
__device__ __forceinline__ int wc_search(const MgTreeNode *__restrict__ T, const MgWorldDesc &W, const int32_t *t, uint64_t &dist,
                                      bool &tied) {
    RtTarget q;
    if (!rt_target(T, t, q) || !rt_packed(T)) return tree_search_tie_stack(T, t, dist, tied);
    const RtWarp r = rt_point(T, W, q, 0xFFFFFFFEu);
    if (r.leaf < 0) return tree_search_tie_stack(T, t, dist, tied);
    dist = r.best;
    tied = r.cnt >= 2;
    return W.leaf_off + r.leaf;
}

/* BiomeManager's cell of block (x, y, z): zoom_cell with one candidate per lane of the first 8 */
__device__ __forceinline__ void wc_zoom(int64_t zseed, int x, int y, int z, int &cx, int &cy, int &cz) {
    const int i = threadIdx.x & 7;
    const int ax = x - 2, ay = y - 2, az = z - 2, px = ax >> 2, py = ay >> 2, pz = az >> 2;
    const int ox = (i >> 2) & 1, oy = (i >> 1) & 1, oz = i & 1;
    const float d = zoom_dist_f(zoom_draws(zseed, px + ox, py + oy, pz + oz), (ax & 3) - 4 * ox, (ay & 3) - 4 * oy, (az & 3) - 4 * oz);
    const float lim = __uint_as_float(__reduce_min_sync(WC_FULL, __float_as_uint(d))) + ZOOM_MARGIN; /* d >= 0: ordered as its bits */
    const unsigned m = __ballot_sync(WC_FULL, d <= lim) & 0xFFu;
    int best = __ffs((int)m) - 1, close;
    if (m & (m - 1)) best = zoom_pick(zseed, px, py, pz, ax & 3, ay & 3, az & 3, close); /* close ones in double precision */
    cx = px + ((best >> 2) & 1);
    cy = py + ((best >> 1) & 1);
    cz = pz + (best & 1);
}

/* cell_chunk (climate.cuh) of one cell, the same in every lane: a tied cell's chain walks back one cell at a time, and after
 * WC_SERIAL cells 32 at a time, a cell per lane (long chains: whole columns at one depth of a flat target). */
#define WC_SERIAL 6
template <bool FM, int DIM>
__device__ __noinline__ int wc_cell_chunk(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                          const MgTreeNode *__restrict__ tree, int qx, int qy, int qz) {
    const int lane = threadIdx.x & 31;
    const int qmin = W.min_y >> 2, qh = W.height >> 2;
    qy = qy < qmin ? qmin : (qy > qmin + qh - 1 ? qmin + qh - 1 : qy);
    int32_t tg0[6], tg[6];
    uint64_t d0, d;
    bool tied;
    wc_target<FM, DIM>(W, S, T, qx, qy, qz, tg0);
    const int leaf0 = wc_search(tree, W, tg0, d0, tied);
    const int bx = qx & ~3, bz = qz & ~3, ly = qy - qmin;
    const int idx0 = (ly >> 2) * 64 + (qx & 3) * 16 + (ly & 3) * 4 + (qz & 3);
    if (idx0 == 0 || !tied) return tree[leaf0].biome;
    /* cell of fill index i */
    auto cx = [&](int i) { return bx + ((i & 63) >> 4); };
    auto cy = [&](int i) { return qmin + (i >> 6) * 4 + (((i & 63) >> 2) & 3); };
    auto cz = [&](int i) { return bz + (i & 3); };
    int idx = idx0 - 1, leaf = -1;
    bool done = false;
    for (int n = 0; n < WC_SERIAL; n++) {
        wc_target<FM, DIM>(W, S, T, cx(idx), cy(idx), cz(idx), tg);
        leaf = wc_search(tree, W, tg, d, tied);
        done = idx == 0 || !tied;
        if (done) break;
        idx--;
    }
    if (!done) { /* still tied: 32 cells a round, a cell per lane, until one of them is untied or first */
        for (;; idx -= 32) {
            const int i = idx - lane;
            bool end = false;
            int l = -1;
            if (i >= 0) {
                cell_target<FM, DIM>(W, S, T, cx(i), cy(i), cz(i), tg);
                l = tree_search_tie(tree, tg, d, tied);
                end = i == 0 || !tied;
            }
            const unsigned m = __ballot_sync(WC_FULL, end);
            if (!m) continue;
            const int j = __ffs((int)m) - 1; /* the nearest one */
            leaf = __shfl_sync(WC_FULL, l, j);
            idx -= j;
            break;
        }
    }
    /* replay the chain forward, 32 cells a round: each lane's target and search, then the candidate in order */
    for (int k0 = idx + 1; k0 < idx0; k0 += 32) {
        const int nk = min(32, idx0 - k0);
        int l = -1;
        uint64_t ld = 0;
        if (nk <= 2) { /* short chains again by the whole warp */
            for (int k = 0; k < nk; k++) {
                wc_target<FM, DIM>(W, S, T, cx(k0 + k), cy(k0 + k), cz(k0 + k), tg);
                const int l0 = wc_search(tree, W, tg, d, tied);
                if (node_dist(tree[leaf], tg) != d) leaf = l0;
            }
            continue;
        }
        if (lane < nk) {
            cell_target<FM, DIM>(W, S, T, cx(k0 + lane), cy(k0 + lane), cz(k0 + lane), tg);
            l = tree_search(tree, tg, -1, ld);
        }
        for (int k = 0; k < nk; k++) { /* lane k's cell keeps the candidate when that is at its minimum too */
            const int l0 = __shfl_sync(WC_FULL, lane < nk && node_dist(tree[leaf], tg) != ld ? l : leaf, k);
            leaf = l0;
        }
    }
    if (node_dist(tree[leaf], tg0) != d0) leaf = leaf0; /* the cell's own step */
    return tree[leaf].biome;
}

/* the same by a block: its warps take the cell and the ones before it at once, one each, so that a chain of up to WB warps'
 * cells (nearly all) costs the time of one; further rounds while it lasts, and past WC_STEPS cells the first warp alone (the
 * walk above).  The result is valid in thread 0; all threads call it, a barrier has to precede the next call. */
#define WC_STEPS 64
struct WcStep {
    int32_t tg[6];
    int32_t leaf, tied;
    uint64_t d;
};
template <bool FM, int DIM, int WB>
__device__ __forceinline__ int wc_block_chunk(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                              const MgTreeNode *__restrict__ tree, int qx, int qy, int qz, WcStep *steps) {
    const int qmin = W.min_y >> 2, qh = W.height >> 2;
    const int y = qy < qmin ? qmin : (qy > qmin + qh - 1 ? qmin + qh - 1 : qy);
    const int bx = qx & ~3, bz = qz & ~3, ly = y - qmin;
    const int idx0 = (ly >> 2) * 64 + (qx & 3) * 16 + (ly & 3) * 4 + (qz & 3);
    for (int s0 = 0; s0 < WC_STEPS; s0 += WB) {
        const int s = s0 + (int)(threadIdx.x >> 5), i = idx0 - s;
        if (i >= 0) {
            int32_t tg[6];
            uint64_t d;
            bool tied;
            wc_target<FM, DIM>(W, S, T, bx + ((i & 63) >> 4), qmin + (i >> 6) * 4 + ((i >> 2) & 3), bz + (i & 3), tg);
            const int leaf = wc_search(tree, W, tg, d, tied);
            if ((threadIdx.x & 31) == 0) {
                for (int k = 0; k < 6; k++) steps[s].tg[k] = tg[k];
                steps[s].leaf = leaf;
                steps[s].tied = tied;
                steps[s].d = d;
            }
        }
        __syncthreads();
        for (int e = s0; e < s0 + WB && e <= idx0; e++) {
            if (steps[e].tied && e < idx0) continue; /* e: the first untied cell back, or the column's first */
            int leaf = steps[e].leaf;
            for (int k = e - 1; k >= 0; k--) /* forward again, the cell itself last */
                if (node_dist(tree[leaf], steps[k].tg) != steps[k].d) leaf = steps[k].leaf;
            return tree[leaf].biome;
        }
    }
    return threadIdx.x < 32 ? wc_cell_chunk<FM, DIM>(W, S, T, tree, qx, qy, qz) : 0;
}

}  // namespace mg
#endif
