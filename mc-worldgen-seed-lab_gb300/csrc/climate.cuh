/* climate.cuh -- climate, End island, zoom and chunk-cell functions of the biome path (device).
 *
 * Shared by the grid/point kernels (kernels.cu) and the fused many-seed kernel (fused.cu).
 */
#ifndef MG_CLIMATE_CUH
#define MG_CLIMATE_CUH
#include "device.cuh"

namespace mg {
using namespace mgd;

/* ============================================================================ climate */
/* ridges_folded, offset spline, y-clamped depth gradient and quantisation of the five noise values
 * (engine/mc_climate.h:126-170), float branch */
__device__ __forceinline__ void climate_finish_f(const MgWorldDesc &W, const MgSpline &S, float tv, float hv, float cv,
                                                 float ev, float rv, int by, int32_t tg[6]) {
    float a = fabsf(rv) + W.rf_f[0];
    float rf = (fabsf(a) + W.rf_f[1]) * W.rf_f[2];
    float co[4] = {cv, ev, rv, rf};
    float off = W.off_f + spline_eval(S, co);
    int lo = min(W.grad_from_y, W.grad_to_y), hi = max(W.grad_from_y, W.grad_to_y);
    int yy = by < lo ? lo : (by > hi ? hi : by);
    float depth = (W.grad_from_f + (float)(yy - W.grad_from_y) * W.grad_fac_f) + off;
    tg[0] = quantize(tv); tg[1] = quantize(hv); tg[2] = quantize(cv);
    tg[3] = quantize(ev); tg[4] = quantize(depth); tg[5] = quantize(rv);
}
/* the double branch's depth gradient at block y, clamped (y_clamped_gradient): a function of y alone, which
 * the tile kernels compute once per tile (an IEEE double division and conversions: about 20 FP64 operations) */
__device__ __forceinline__ double depth_grad_d(const MgWorldDesc &W, int by) {
    const double fac = ((double)by - (double)W.grad_from_y) / ((double)W.grad_to_y - (double)W.grad_from_y);
    return fac < 0.0 ? W.grad_from_d : (fac > 1.0 ? W.grad_to_d : W.grad_from_d + fac * (W.grad_to_d - W.grad_from_d));
}
/* the same in the double branch */
__device__ __forceinline__ void climate_finish_d(const MgWorldDesc &W, const MgSpline &S, double tv, double hv, double cv,
                                                 double ev, double rv, int by, int32_t tg[6]) {
    double rf = (fabs(fabs(rv) + W.rf_d[0]) + W.rf_d[1]) * W.rf_d[2];
    float co[4] = {(float)cv, (float)ev, (float)rv, (float)rf};
    double off = 0.0 + (W.off_d + (double)spline_eval(S, co)) * 1.0;
    double depth = depth_grad_d(W, by) + off;
    tg[0] = quantize((float)tv); tg[1] = quantize((float)hv); tg[2] = quantize((float)cv);
    tg[3] = quantize((float)ev); tg[4] = quantize((float)depth); tg[5] = quantize((float)rv);
}

/* the same from the float values the reference takes of the five noises and of ridges_folded, with the
 * depth gradient g = depth_grad_d(W, by) given */
__device__ __forceinline__ void climate_finish_df(const MgWorldDesc &W, const MgSpline &S, float tf, float hf, float cf,
                                                  float ef, float rvf, float rff, double g, int32_t tg[6]) {
    float co[4] = {cf, ef, rvf, rff};
    double off = 0.0 + (W.off_d + (double)spline_eval(S, co)) * 1.0;
    double depth = g + off;
    tg[0] = quantize(tf); tg[1] = quantize(hf); tg[2] = quantize(cf);
    tg[3] = quantize(ef); tg[4] = quantize((float)depth); tg[5] = quantize(rvf);
}
/* (float) of a double-branch NormalNoise at (x, 0, z): the screened fixed-point value when it settles the
 * rounding, else the exact double evaluation */
__device__ __forceinline__ float nn_d_y0_float(const MgNoise &N, const MgLattice *__restrict__ T, double x, double z,
                                               double xc, double zc) {
    float f;
    if (N.fix_eq >= 0) {
        const int64_t q = nn_q<false>(N, T, x, z, xc, zc);
        if (q != MG_QFAIL && cast_settled_q(q, N.fix_eq, f)) return f;
    }
    return (float)nn_d_y0(N, T, x, z, xc, zc);
}
/* a value only quantised, from a fixed-point approximation q (units of 2^-59) within eq units of the
 * reference's double value v: true when every real in [q - eq, q + eq] 2^-59 has the target of the two ends
 * (the rounding to float, the product by 10000 and the truncation are each monotone, so the ends settle
 * quantize((float)v)); f is then a float with that target (the lower end's) */
__device__ __forceinline__ bool quant_settled_q(int64_t q, int64_t eq, float &f) {
    const float lo = __ll2float_rn(q - eq) * 0x1.0p-59f, hi = __ll2float_rn(q + eq) * 0x1.0p-59f;
    f = lo;
    return quantize(lo) == quantize(hi);
}
/* a float with the target of a double-branch NormalNoise's value at (x, 0, z), for a noise whose float is
 * only quantised (the Nether's two): the 32-bit screen's when it settles the target, else nn_d_y0_float's
 * (the float itself).  The Overworld's temperature and vegetation are only quantised too, but there the
 * second octave form measured slower: its code pushed the double branch's hot path out of the instruction
 * cache. */
__device__ __forceinline__ float nn_d_y0_qfloat(const MgNoise &N, const MgLattice *__restrict__ T, double x, double z,
                                                double xc, double zc) {
    float f;
    if (N.fix_eq32 >= 0) {
        const int64_t q = nn_q32(N, T, x, z, xc, zc);
        if (q != MG_QFAIL && quant_settled_q(q, N.fix_eq32, f)) return f;
    }
    return nn_d_y0_float(N, T, x, z, xc, zc);
}
/* ridges_folded (|(|r| + c0)| + c1) * c2 of a ridge value (the exact path) */
__device__ __forceinline__ double ridges_folded_d(const MgWorldDesc &W, double r) {
    return (fabs(fabs(r) + W.rf_d[0]) + W.rf_d[1]) * W.rf_d[2];
}
/* the float of ridges_folded from a fixed-point ridge value q (units of 2^-59) within the ridge screen's
 * bound: the constants are multiples of 2^-59 (W.rf_eq >= 0), so the sums are exact and the product rounds
 * down by less than one unit (it runs for sums below 4; others go to the exact path).  ridges_folded of two
 * values within d of each other differ by at most |c2| d, and the reference's three roundings of it (values
 * below 17) by less than |c2| 1e-14 + 1e-13, so W.rf_eq is |c2| (err + 1e-14) + 1e-13 plus one unit. */
__device__ __forceinline__ bool ridges_folded_settled(const MgWorldDesc &W, int64_t q, float &f) {
    int64_t v = (q < 0 ? -q : q) + W.rf_q[0];
    v = (v < 0 ? -v : v) + W.rf_q[1];
    if (v >= (4LL << MG_Q) || v <= -(4LL << MG_Q)) return false;
    const int64_t c = W.rf_q[2], m = mulq_us(c < 0 ? -c : c, v);
    return cast_settled_q(c < 0 ? -m : m, W.rf_eq, f);
}
/* ridge noise and ridges_folded as floats */
__device__ __forceinline__ void ridge_float(const MgWorldDesc &W, const MgLattice *__restrict__ T, double x, double z,
                                            double xc, double zc, float &rvf, float &rff) {
    const MgNoise &N = W.noise[5];
    if (W.rf_eq >= 0) {
        const int64_t q = nn_q<false>(N, T, x, z, xc, zc);
        if (q != MG_QFAIL && cast_settled_q(q, N.fix_eq, rvf) && ridges_folded_settled(W, q, rff))
            return;
    }
    const double rv = nn_d_y0(N, T, x, z, xc, zc);
    rvf = (float)rv;
    rff = (float)ridges_folded_d(W, rv);
}

/* double branch of the Overworld climate after the shift: the climate noises screened at the exact shifted
 * coordinates, the finish (out of line: reached from the per-cell and the per-tile shift forms) */
static __device__ __noinline__ void climate_ow_d_rest(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                                      double x, double z, double g, int32_t *tg) {
    const double xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
    const float tf = nn_d_y0_float(W.noise[1], T, x, z, xc, zc);
    const float hf = nn_d_y0_float(W.noise[2], T, x, z, xc, zc);
    const float cf = nn_d_y0_float(W.noise[3], T, x, z, xc, zc);
    const float ef = nn_d_y0_float(W.noise[4], T, x, z, xc, zc);
    float rvf, rff;
    ridge_float(W, T, x, z, xc, zc, rvf, rff);
    climate_finish_df(W, S, tf, hf, cf, ef, rvf, rff, g, tg);
}
/* double branch of the Overworld climate, out of line (the kernels reach the climate from two sites each:
 * the cell itself and the tie chain).  The shift noises stay exact in double: their value moves the climate
 * noises' input coordinates, and the kernels' integer pipes (which carry the screened climate noises) are
 * busier than the FP64 pipe, so a fixed-point shift measured slower. */
static __device__ __noinline__ void climate_ow_d(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                                 double X, double Z, double Xc, double Zc, int by, int32_t *tg) {
    const double sx = nn_d_y0(W.noise[0], T, X, Z, Xc, Zc) * 4.0;
    const double sz = nn_d_z0(W.noise[0], T, Z, X, Zc, Xc) * 4.0;
    climate_ow_d_rest(W, S, T, X + sx, Z + sz, depth_grad_d(W, by), tg);
}

/* Overworld climate of quart cell (qx, qy, qz) -> 6 quantised targets (engine/mc_climate.h:113-170). */
template <bool FM>
__device__ __forceinline__ void climate_ow(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                           int qx, int qy, int qz, int32_t tg[6]) {
    const double X = (double)qx, Z = (double)qz; /* blockX * 0.25 with blockX = 4 qx */
    const double Xc = X * MG_SECOND_STACK, Zc = Z * MG_SECOND_STACK;
    const int by = qy * 4;
    if (FM) {
        float sx = nn_f_y0(W.noise[0], T, X, Z, Xc, Zc) * 4.0f; /* ShiftA (x, 0, z) */
        float sz = nn_f_z0(W.noise[0], T, Z, X, Zc, Xc) * 4.0f; /* ShiftB (z, x, 0) */
        double x = X + (double)sx, z = Z + (double)sz;
        double xc = x * MG_SECOND_STACK, zc = z * MG_SECOND_STACK;
        float tv = nn_f_y0(W.noise[1], T, x, z, xc, zc);
        float hv = nn_f_y0(W.noise[2], T, x, z, xc, zc);
        float cv = nn_f_y0(W.noise[3], T, x, z, xc, zc);
        float ev = nn_f_y0(W.noise[4], T, x, z, xc, zc);
        float rv = nn_f_y0(W.noise[5], T, x, z, xc, zc);
        climate_finish_f(W, S, tv, hv, cv, ev, rv, by, tg);
    } else {
        climate_ow_d(W, S, T, X, Z, Xc, Zc, by, tg);
    }
}
/* Nether: temperature and vegetation at (x/4, 0, z/4) (engine/cuda/mcg_host.c:63-74) */
template <bool FM>
__device__ __forceinline__ void climate_nether(const MgWorldDesc &W, const MgLattice *__restrict__ T, int qx, int qz,
                                               int32_t tg[6]) {
    const double X = (double)qx, Z = (double)qz;
    const double Xc = X * MG_SECOND_STACK, Zc = Z * MG_SECOND_STACK;
    float t, h;
    if (FM) {
        t = nn_f_legacy_y0(W.nether[0], T, X, Z, Xc, Zc);
        h = nn_f_legacy_y0(W.nether[1], T, X, Z, Xc, Zc);
    } else {
        t = nn_d_y0_qfloat(W.nether[0], T, X, Z, Xc, Zc);
        h = nn_d_y0_qfloat(W.nether[1], T, X, Z, Xc, Zc);
    }
    tg[0] = quantize(t);
    tg[1] = quantize(h);
    tg[2] = tg[3] = tg[4] = tg[5] = 0;
}
template <bool FM, int DIM>
__device__ __forceinline__ void cell_target(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                            int qx, int qy, int qz, int32_t tg[6]) {
    if (DIM == MG_OVERWORLD) climate_ow<FM>(W, S, T, qx, qy, qz, tg);
    else climate_nether<FM>(W, T, qx, qz, tg);
}

/* ============================================================================ End islands (engine/mc_end.h) */
__device__ __forceinline__ double simplex2(const uint8_t *__restrict__ p, double xin, double yin, double F2, double G2) {
    double s = (xin + yin) * F2;
    int i = ifloor(xin + s), j = ifloor(yin + s);
    double t = (double)(i + j) * G2;
    double x0 = xin - ((double)i - t), y0 = yin - ((double)j - t);
    int i1 = x0 > y0 ? 1 : 0, j1 = 1 - i1;
    double x1 = x0 - (double)i1 + G2, y1 = y0 - (double)j1 + G2;
    double x2 = x0 - 1.0 + 2.0 * G2, y2 = y0 - 1.0 + 2.0 * G2;
    int ii = i & 255, jj = j & 255;
    int g0 = p[(ii + p[jj]) & 255] % 12;
    int g1 = p[(ii + i1 + p[(jj + j1) & 255]) & 255] % 12;
    int g2 = p[(ii + 1 + p[(jj + 1) & 255]) & 255] % 12;
    double n = 0.0, acc[3];
    const double xs[3] = {x0, x1, x2}, ys[3] = {y0, y1, y2};
    const int gs[3] = {g0, g1, g2};
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double tt = 0.5 - xs[c] * xs[c] - ys[c] * ys[c] - 0.0 * 0.0;
        if (tt < 0.0) acc[c] = 0.0;
        else {
            tt *= tt;
            acc[c] = tt * tt * gdot<double>(gs[c], xs[c], ys[c], 0.0);
        }
    }
    n = acc[0] + acc[1] + acc[2];
    return 70.0 * n;
}
/* End island test, screened: the reference decides an island cell by nv < -0.9f (double branch, the float
 * constant widened) or (float)nv < -0.9f (float branch), nv = simplex2 in double (about 60 FP64-pipe
 * operations).  Here the three corner terms are evaluated in float from the first corner's offsets x0, y0:
 * |float value - nv| <= END_ISLAND_E (a forward error bound: offsets within 5 u of the
 * double ones, u = 2^-24; tt = 0.5 - x^2 - y^2 within 32 u; tt^4 within 18 u; the gradient dot within 12 u;
 * each term tt^4 * dot within 26 u for |x|, |y| < 0.71 (tt > 0); three terms and their sums within 78 u; times
 * 70: 5,500 u = 3.3e-4 plus the reference's own double roundings, taken as 5e-4).  A value farther than that
 * from the threshold settles the test (with one more float ulp for the float branch's rounding); the rest
 * (a few in 10^4) take the exact double evaluation.  mcgen_gb300_check_end checks the bound and the decisions
 * on the device.
 *
 * The coordinates are whole numbers, so within END_FAR the skew is fixed point (2^-40) in place of the reference's doubles
 * (9 FP64 operations): x0, y0 come within 3 u (G2's rounding, up to 2^-41 a cell, is added back in float).  Where the cell or the
 * corner choice is nearly ambiguous it may be the reference's neighbour; the corners that the two choices do not share are then
 * at the edge of their terms' support (tt <= 2e-6, cut off at 0), so the value is within the bound all the same. */
#define END_ISLAND_E 5e-4f
#define END_FAR (1 << 21)
#define END_Q 40
#define END_F2Q ((int64_t)(0.36602540378443865 * (double)(1LL << END_Q)))
#define END_G2Q ((int64_t)(0.21132486540518713 * (double)(1LL << END_Q)))
struct EndCell {
    int i, j;
    float x0, y0;
};
/* |tx|, |tz| < END_FAR */
__device__ __forceinline__ EndCell end_cell(int tx, int tz, double G2) {
    const float g2e = (float)(G2 - (double)END_G2Q * 0x1.0p-40);
    const int64_t s = (int64_t)(tx + tz) * END_F2Q;
    EndCell c;
    c.i = (int)((((int64_t)tx << END_Q) + s) >> END_Q);
    c.j = (int)((((int64_t)tz << END_Q) + s) >> END_Q);
    const int64_t t = (int64_t)(c.i + c.j) * END_G2Q;
    const float te = (float)(c.i + c.j) * g2e;
    c.x0 = (float)(int32_t)((((int64_t)(tx - c.i) << END_Q) + t) >> 10) * 0x1.0p-30f + te;
    c.y0 = (float)(int32_t)((((int64_t)(tz - c.j) << END_Q) + t) >> 10) * 0x1.0p-30f + te;
    return c;
}
/* the gradient of a permutation value, its third component dropped */
__device__ __forceinline__ float2 end_grad(int v) {
    const int g = v % 12;
    return make_float2(gdot<float>(g, 1.0f, 0.0f, 0.0f), gdot<float>(g, 0.0f, 1.0f, 0.0f));
}
/* the three terms times 70; G(k): the gradient of p[k] */
template <typename GRAD>
__device__ __forceinline__ float end_simplex_f(const uint8_t *__restrict__ p, const GRAD &G, const EndCell &e, float g2) {
    const int i1 = e.x0 > e.y0 ? 1 : 0, j1 = 1 - i1;
    const float xs[3] = {e.x0, e.x0 - (float)i1 + g2, e.x0 - 1.0f + 2.0f * g2};
    const float ys[3] = {e.y0, e.y0 - (float)j1 + g2, e.y0 - 1.0f + 2.0f * g2};
    const int ii = e.i & 255, jj = e.j & 255;
    const float2 gs[3] = {G((ii + p[jj]) & 255), G((ii + i1 + p[(jj + j1) & 255]) & 255), G((ii + 1 + p[(jj + 1) & 255]) & 255)};
    float n = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        float tt = fmaxf(0.5f - xs[c] * xs[c] - ys[c] * ys[c], 0.0f);
        tt *= tt;
        n += tt * tt * (gs[c].x * xs[c] + gs[c].y * ys[c]);
    }
    return n * 70.0f;
}
template <typename GRAD>
__device__ __forceinline__ bool end_island_g(const uint8_t *__restrict__ p, const GRAD &G, long long tx, long long tz, double F2, double G2,
                                             bool fm) {
    EndCell e;
    if (tx > -END_FAR && tx < END_FAR && tz > -END_FAR && tz < END_FAR) {
        e = end_cell((int)tx, (int)tz, G2);
    } else {
        const double xin = (double)tx, yin = (double)tz, s = (xin + yin) * F2;
        e.i = ifloor(xin + s);
        e.j = ifloor(yin + s);
        const double t = (double)(e.i + e.j) * G2;
        e.x0 = (float)(xin - ((double)e.i - t));
        e.y0 = (float)(yin - ((double)e.j - t));
    }
    const float n = end_simplex_f(p, G, e, (float)G2);
    if (fabsf(n + 0.9f) > END_ISLAND_E + 1e-4f) return n < -0.9f;
    const double nv = simplex2(p, (double)tx, (double)tz, F2, G2);
    return fm ? ((float)nv < -0.9f) : (nv < (double)-0.9f);
}
__device__ __forceinline__ bool end_island(const uint8_t *__restrict__ p, long long tx, long long tz, double F2, double G2, bool fm) {
    return end_island_g(p, [&](int k) { return end_grad(p[k]); }, tx, tz, F2, G2, fm);
}
/* (float)sqrt((double)v): rounding the double root to float is the float root correctly rounded, since a double has more than
 * twice a float's bits plus two; the double root costs 20 operations of the FP64 pipe */
__device__ __forceinline__ float end_sqrt(float v) { return __fsqrt_rn(v); }
/* island size fmod(|x| 3439 + |z| 147, 13) + 9: the sum is a whole number (its parts are, rounded or not), below 2^32 within
 * 1.2 million chunk cells */
__device__ __forceinline__ float end_size(float tx, float tz) {
    const float a = fabsf(tx) * 3439.0f + fabsf(tz) * 147.0f;
    if (a < 4294967040.0f) return (float)((uint32_t)a % 13u) + 9.0f;
    return fmodf(a, 13.0f) + 9.0f;
}
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return v < lo ? lo : (v < hi ? v : hi); }
/* EndIslandDensityFunction.getHeightValue at (sx, sz) = (block / 8) by a warp (all 32 lanes call it, the same result): the 25 x 25
 * island cells over the lanes.  One thread took 700 us for a chunk's 625 cells. */
inline __device__ float end_height(const uint8_t *__restrict__ p, bool fm, int sx, int sz, double F2, double G2) {
    int cx = sx / 2, cz = sz / 2, ox = sx % 2, oz = sz % 2;
    float best;
    if (!fm) {
        int32_t sq = (int32_t)((uint32_t)sx * (uint32_t)sx + (uint32_t)sz * (uint32_t)sz); /* Java int overflow */
        float len = end_sqrt((float)sq);
        best = clampf(100.0f - len * 8.0f, -100.0f, 80.0f);
    } else best = -100.0f;
    for (int k = threadIdx.x & 31; k < 625; k += 32) {
        const int dx = k % 25 - 12, dz = k / 25 - 12;
        long long tx = (long long)cx + dx, tz = (long long)cz + dz;
        if (tx * tx + tz * tz <= 4096LL) continue;
        if (!end_island(p, tx, tz, F2, G2, fm)) continue;
        float size = end_size((float)tx, (float)tz);
        float xd = (float)(ox - dx * 2), zd = (float)(oz - dz * 2);
        float h = clampf(100.0f - end_sqrt(xd * xd + zd * zd) * size, -100.0f, 80.0f);
        best = best > h ? best : h;
    }
    for (int d = 16; d; d >>= 1) {
        const float o = __shfl_xor_sync(0xFFFFFFFFu, best, d);
        best = best > o ? best : o;
    }
    return best;
}
/* TheEndBiomeSource class of chunk (cx, cz): 0 the_end, 1 highlands, 2 midlands, 3 small islands, 4 barrens; by a warp, like
 * end_height */
inline __device__ int end_chunk_class(const uint8_t *__restrict__ p, bool fm, int cx, int cz, double F2, double G2) {
    if ((long long)cx * cx + (long long)cz * cz <= 4096LL) return 0;
    int bx = (cx * 2 + 1) * 8, bz = (cz * 2 + 1) * 8;
    float h = end_height(p, fm, bx / 8, bz / 8, F2, G2);
    double e;
    if (!fm) e = ((double)h - 8.0) / 128.0;
    else {
        float dx = (float)(0 - bx), dz = (float)(0 - bz);
        float len = end_sqrt(dx * dx + 0.0f * 0.0f + dz * dz);
        float c = (clampf(100.0f - len, -100.0f, 80.0f) - 8.0f) * 0.0078125f;
        float o = (h - 8.0f) / 128.0f;
        e = (double)(c > o ? c : o);
    }
    if (e > 0.25) return 1;
    if (e >= -0.0625) return 2;
    return e < -0.21875 ? 3 : 4;
}

/* ---------------------------------------------------------------------------- BiomeManager zoom
 * (libmcgen/src/region.c:61-85) */
__device__ __forceinline__ int64_t zoom_step(int64_t r, int64_t c) {
    uint64_t v = (uint64_t)r;
    v *= v * 6364136223846793005ULL + 1442695040888963407ULL;
    return (int64_t)(v + (uint64_t)c);
}
/* Math.floorMod(r >> 24, 1024) / 1024.0: the ten bits above bit 23; the division by 2^10 is exact as a scaling */
__device__ __forceinline__ int zoom_bits(int64_t r) { return (int)((r >> 24) & 1023); }
__device__ __forceinline__ double zoom_jitter(int m) { return ((double)m * 0x1.0p-10 - 0.5) * 0.9; }
/* the three jitter draws of candidate cell (x, y, z), ten bits each (x in bits 0-9, y 10-19, z 20-29) */
__device__ __forceinline__ uint32_t zoom_draws(int64_t seed, int x, int y, int z) {
    int64_t r = seed;
    r = zoom_step(r, x); r = zoom_step(r, y); r = zoom_step(r, z);
    r = zoom_step(r, x); r = zoom_step(r, y); r = zoom_step(r, z);
    uint32_t m = (uint32_t)zoom_bits(r);
    r = zoom_step(r, seed);
    m |= (uint32_t)zoom_bits(r) << 10;
    r = zoom_step(r, seed);
    return m | (uint32_t)zoom_bits(r) << 20;
}
/* the fiddled distance in double, in the reference's order (z, y, x terms) */
__device__ __forceinline__ double zoom_dist_d(uint32_t m, double dx, double dy, double dz) {
    const double jx = zoom_jitter((int)(m & 1023)), jy = zoom_jitter((int)((m >> 10) & 1023)),
                 jz = zoom_jitter((int)(m >> 20));
    return (dz + jz) * (dz + jz) + (dy + jy) * (dy + jy) + (dx + jx) * (dx + jx);
}
/* The same in single precision, as a screen.  Against the double value it differs by at most 1.23e-6: each
 * of the three squared terms by at most 2.48e-7 (the maximum over all 8 x 1024 (offset, draw) pairs, the
 * draw's jitter taken as (m - 512) * fl32(0.9 / 1024)), and the two single-precision additions of terms below
 * 6.31 by half an ulp (2^-22) each.  So a candidate whose screened distance exceeds the smallest screened one
 * by more than ZOOM_MARGIN (four times twice that bound) cannot be the double-precision minimum. */
#define ZOOM_MARGIN 1e-5f
__device__ __forceinline__ float zoom_dist_f(uint32_t m, int qx, int qy, int qz) {
    const float c = 0.9f / 1024.0f;
    const float ux = (float)qx * 0.25f + (float)((int)(m & 1023) - 512) * c;
    const float uy = (float)qy * 0.25f + (float)((int)((m >> 10) & 1023) - 512) * c;
    const float uz = (float)qz * 0.25f + (float)((int)(m >> 20) - 512) * c;
    return uz * uz + uy * uy + ux * ux;
}
/* BiomeManager.getBiome's choice among the 8 quart cells around block (x, y, z): the first candidate (in the
 * order x, y, z bit = 0 first) with the smallest double-precision fiddled distance.  The distances are
 * screened in single precision; only when a second candidate lies within ZOOM_MARGIN of the smallest are the
 * close candidates' distances taken in double precision (in candidate order, strict comparison), which
 * gives the same choice as the double-precision comparison of all 8. */
__device__ __forceinline__ int zoom_pick(int64_t zseed, int px, int py, int pz, int fx, int fy, int fz, int &close) {
    uint32_t mm[8];
    float df[8];
    float bf = __int_as_float(0x7F800000);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int ox = (i >> 2) & 1, oy = (i >> 1) & 1, oz = i & 1;
        mm[i] = zoom_draws(zseed, px + ox, py + oy, pz + oz);
        df[i] = zoom_dist_f(mm[i], fx - 4 * ox, fy - 4 * oy, fz - 4 * oz);
        bf = fminf(bf, df[i]);
    }
    const float lim = bf + ZOOM_MARGIN;
    int best = -1;
    close = 0;
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (df[i] <= lim) { close++; if (best < 0) best = i; }
    if (close > 1) {
        double bd = __longlong_as_double(0x7FF0000000000000LL);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (df[i] > lim) continue;
            const int ox = (i >> 2) & 1, oy = (i >> 1) & 1, oz = i & 1;
            const double d = zoom_dist_d(mm[i], fx * 0.25 - ox, fy * 0.25 - oy, fz * 0.25 - oz);
            if (bd > d) { best = i; bd = d; }
        }
    }
    return best;
}
__device__ __forceinline__ void zoom_cell(int64_t zseed, int x, int y, int z, int &cx, int &cy, int &cz) {
    const int ax = x - 2, ay = y - 2, az = z - 2;
    const int px = ax >> 2, py = ay >> 2, pz = az >> 2;
    int close;
    const int best = zoom_pick(zseed, px, py, pz, ax & 3, ay & 3, az & 3, close);
    cx = px + ((best >> 2) & 1);
    cy = py + ((best >> 1) & 1);
    cz = pz + (best & 1);
}
/* The chain of cell_chunk, given the cell's own target tg0 and search (leaf0, the first leaf at the minimum
 * distance d0, and whether another leaf ties it): when the cell is tied, walk back to the first untied cell of
 * the chunk's fill order and replay the chain forward, the cell's own step from tg0, leaf0 and d0 (a tied
 * lane pays one climate evaluation per cell walked back, not two; its warp waits for it). */
template <bool FM, int DIM>
__device__ int cell_chunk_chain(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                const MgTreeNode *__restrict__ tree, int qx, int qy, int qz, const int32_t *tg0,
                                int leaf0, uint64_t d0, bool tied) {
    const int qmin = W.min_y >> 2, qh = W.height >> 2;
    qy = qy < qmin ? qmin : (qy > qmin + qh - 1 ? qmin + qh - 1 : qy);
    const int bx = qx & ~3, bz = qz & ~3, ly = qy - qmin;
    const int idx0 = (ly >> 2) * 64 + (qx & 3) * 16 + (ly & 3) * 4 + (qz & 3);
    if (idx0 == 0 || !tied) return tree[leaf0].biome;
    int32_t tg[6];
    uint64_t d;
    int idx = idx0 - 1, leaf;
    for (;;) {
        int sec = idx >> 6, r = idx & 63;
        cell_target<FM, DIM>(W, S, T, bx + (r >> 4), qmin + sec * 4 + ((r >> 2) & 3), bz + (r & 3), tg);
        leaf = tree_search_tie(tree, tg, d, tied);
        if (idx == 0 || !tied) break;
        idx--;
    }
    for (int k = idx + 1; k < idx0; k++) { /* replay the chain forward */
        int sec = k >> 6, r = k & 63;
        cell_target<FM, DIM>(W, S, T, bx + (r >> 4), qmin + sec * 4 + ((r >> 2) & 3), bz + (r & 3), tg);
        int l0 = tree_search(tree, tg, -1, d);
        if (node_dist(tree[leaf], tg) != d) leaf = l0;
    }
    if (node_dist(tree[leaf], tg0) != d0) leaf = leaf0; /* the cell's own step */
    return tree[leaf].biome;
}
/* world_biome_cell (libmcgen/src/biome.c:87-114): y clamped into the dimension; a tied cell walks back along
 * LevelChunkSection.fillBiomesFromNoise order (sections bottom-up, then x, y, z) to an untied cell or the
 * column's first cell, then replays the candidate chain forward.  The walk is bounded by the column.  Out of
 * line: the batch kernel reaches it only for requests under this rule, and inlined its code and registers
 * weighed on the other paths' hot code (spills and the instruction cache). */
template <bool FM, int DIM>
__device__ __noinline__ int cell_chunk(const MgWorldDesc &W, const MgSpline &S, const MgLattice *__restrict__ T,
                                       const MgTreeNode *__restrict__ tree, int qx, int qy, int qz) {
    const int qmin = W.min_y >> 2, qh = W.height >> 2;
    const int cy = qy < qmin ? qmin : (qy > qmin + qh - 1 ? qmin + qh - 1 : qy);
    int32_t tg[6];
    cell_target<FM, DIM>(W, S, T, qx, cy, qz, tg);
    uint64_t d;
    bool tied;
    const int leaf = tree_search_tie(tree, tg, d, tied);
    return cell_chunk_chain<FM, DIM>(W, S, T, tree, qx, qy, qz, tg, leaf, d, tied);
}

}  // namespace mg
#endif
