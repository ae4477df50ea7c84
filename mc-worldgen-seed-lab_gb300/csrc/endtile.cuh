/* endtile.cuh -- End island classes of a tile of chunks, shared by the batched kernel and the plain
 * per-request End path.
 *
 * TheEndBiomeSource's class of chunk c needs the island field at the 25 x 25 chunk cells around c
 * (engine/mc_end.h:66-119).  A tile of w x h chunks evaluates the simplex field once over its (w + 24) x (h + 24)-cell window,
 * kept as a mask of islands per row, instead of 625 times per chunk; then a thread per chunk visits only the island bits of its 25
 * rows (the maximum does not depend on the order).  Up to 24 x 24 chunks: 4 cells a chunk, where 8 x 8 took 16, and a grid is cut
 * into equal tiles (17 chunks: one of 17, not three of 8 whose windows overlap).
 *
 * 4,096 requests of 64 x 64 cells: 2,270 us with end_island's skew and the heights' roots in double and 8 x 8 tiles (17,800
 * cycles per tile, most of them FP64), 148 us so. */
#ifndef MG_ENDTILE_CUH
#define MG_ENDTILE_CUH
#include "climate.cuh"

namespace mg {

#define END_TC 24 /* chunks per End tile side, at most */
#define END_WIN (END_TC + 24)

struct EndTile {
    uint64_t rows[END_WIN];              /* bit i of rows[r]: window cell (i, r) is an island */
    float2 grad[256];                    /* gradient of p[k] (end_tile_grad) */
    uint8_t isize[END_WIN * END_WIN];    /* its size */
    uint8_t cls[END_TC * END_TC];        /* class of tile chunk (cx0 + i % w, cz0 + i / w) */
};

/* the side of the equal tiles that n chunks are cut into, each at most cap */
__host__ __device__ inline int end_tile_side(int n, int cap) {
    const int tiles = (n + cap - 1) / cap;
    return (n + tiles - 1) / tiles;
}
/* the gradients of a permutation, by a block (a barrier has to follow) */
__device__ __forceinline__ void end_tile_grad(const uint8_t *p, EndTile &e) {
    for (int k = threadIdx.x; k < 256; k += blockDim.x) e.grad[k] = end_grad(p[k]);
}
/* classes of chunks [cx0, cx0 + w) x [cz0, cz0 + h) into e.cls; p: the End simplex permutation, its gradients in e.grad */
template <bool FM>
__device__ __forceinline__ void end_tile_classes(const uint8_t *__restrict__ p, double F2, double G2, int cx0, int cz0, int w, int h,
                                                 EndTile &e) {
    /* chunk c's height reads chunk cells c' + d, d in [-12, 12], with c' = (2c+1)/2 in Java int division
     * (c for c >= 0, c + 1 for c < 0): a window of at most w - 1 + 25 cells per axis */
    const int wx0 = (cx0 * 2 + 1) / 2 - 12, wz0 = (cz0 * 2 + 1) / 2 - 12;
    const int lane = threadIdx.x & 31;
    uint32_t *half_rows = reinterpret_cast<uint32_t *>(e.rows);
    for (int u = threadIdx.x >> 5; u < 2 * (h + 24); u += (int)(blockDim.x >> 5)) { /* half a window row per warp */
        const int r = u >> 1, c = (u & 1) * 32 + lane;
        const int tx = wx0 + c, tz = wz0 + r;
        bool isl = false;
        if (c < w + 24 && (long long)tx * tx + (long long)tz * tz > 4096LL) {
            isl = end_island_g(p, [&](int k) { return e.grad[k]; }, tx, tz, F2, G2, FM);
            if (isl) e.isize[r * END_WIN + c] = (uint8_t)end_size((float)tx, (float)tz);
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, isl);
        if (lane == 0) half_rows[u] = m;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < w * h; c += blockDim.x) {
        const int cx = cx0 + c % w, cz = cz0 + c / w;
        int cls = 0;
        if ((long long)cx * cx + (long long)cz * cz > 4096LL) {
            const int bx = (cx * 2 + 1) * 8, bz = (cz * 2 + 1) * 8;
            const int sx = bx / 8, sz = bz / 8;
            const int ccx = sx / 2, ccz = sz / 2, ox = sx % 2, oz = sz % 2;
            float best = -100.0f;
            if (!FM) {
                int32_t sq = (int32_t)((uint32_t)sx * (uint32_t)sx + (uint32_t)sz * (uint32_t)sz);
                best = clampf(100.0f - end_sqrt((float)sq) * 8.0f, -100.0f, 80.0f);
            }
            const int sh = ccx - 12 - wx0; /* 0 .. w - 1 */
            for (int dz = -12; dz <= 12; dz++) {
                const int row = ccz + dz - wz0;
                uint32_t m = (uint32_t)(e.rows[row] >> sh) & 0x1FFFFFFu;
                while (m) {
                    const int b = __ffs((int)m) - 1;
                    m &= m - 1;
                    const float xd = (float)(ox - (b - 12) * 2), zd = (float)(oz - dz * 2);
                    const float hh = clampf(100.0f - end_sqrt(xd * xd + zd * zd) * (float)e.isize[row * END_WIN + b + sh], -100.0f, 80.0f);
                    best = best > hh ? best : hh;
                }
            }
            double ev;
            if (!FM) ev = ((double)best - 8.0) / 128.0;
            else {
                const float ddx = (float)(0 - bx), ddz = (float)(0 - bz);
                const float len = end_sqrt(ddx * ddx + 0.0f * 0.0f + ddz * ddz);
                const float cc = (clampf(100.0f - len, -100.0f, 80.0f) - 8.0f) * 0.0078125f;
                const float o = (best - 8.0f) / 128.0f;
                ev = (double)(cc > o ? cc : o);
            }
            cls = ev > 0.25 ? 1 : (ev >= -0.0625 ? 2 : (ev < -0.21875 ? 3 : 4));
        }
        e.cls[c] = (uint8_t)cls;
    }
    __syncthreads();
}

}  // namespace mg
#endif
