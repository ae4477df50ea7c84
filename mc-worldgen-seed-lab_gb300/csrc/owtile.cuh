/* owtile.cuh -- Overworld climate of a 16 x 16-cell tile from tables of lattice nodes (device).
 *
 * Every NormalNoise on the biome path has one input coordinate that is zero, so an octave is a function of two
 * coordinates over a plane of its lattice, and a tile of neighbouring cells touches few of the plane's nodes:
 * 4 to 9 for the octaves below 2^-5 per quart (32 of the climate's 40), about 150 for the finest one.  The
 * per-cell forms (device.cuh octave_q) look up 14 permutation bytes and 8 gradients per octave sample, which is
 * most of their time.  Here the CTA builds the nodes once per tile (two gradients of a node: the two lattice
 * planes around the zero coordinate's fixed offset) into shared memory, and a cell reads its four nodes.
 *
 * Phases of a tile (256 threads, one cell each, warps of 8 x 4 cells):
 *   1  the shift noises' splits per column and row, and their nodes (the inputs are the integer quart grid)
 *   2  per cell: both shift noises, the shifted coordinates, and their range over the tile
 *   3  one warp: each climate octave's node range and place in the table; another takes the next tile
 *   4  the climate octaves' nodes
 *   5  per cell: the climate noises and what follows from them
 */
#ifndef MG_OWTILE_CUH
#define MG_OWTILE_CUH
#include "climate.cuh"

namespace mg {

#define OT_W 16                   /* tile width and height in cells */
#define OT_TABW 17                /* quart columns a tile's cells may lie in (BiomeManager's zoom of blocks up to 4 apart: one more) */
#define OT_NT (OT_W * OT_W)       /* threads per CTA */
#define OT_MAXLEV 3               /* levels of the shift noise (26.x: 3) */
#define OT_SHIFT_TABS (4 * OT_MAXLEV)
#define OT_DEPTH_LIM 3.0          /* |depth gradient + offset constant|, for the depth in units of 2^-28 */
#define OT_COORD_LIM ((1 << 23) - 4096) /* |quart| below which every wrap of the path is the identity */

/* column and row of this thread's cell: warps take 8 x 4 blocks, so the R-tree walk of a warp has a compact box */
__device__ __forceinline__ int ot_col() { return ((threadIdx.x >> 5) & 1) * 8 + (threadIdx.x & 7); }
__device__ __forceinline__ int ot_row() { return (threadIdx.x >> 6) * 4 + ((threadIdx.x >> 3) & 3); }

/* nodes per axis that OT_TABW neighbouring quart columns can touch at frequency f (second stack: 1.0181... f) */
__host__ __device__ inline int ot_shift_nodes(double f) { return (int)((OT_TABW - 1) * f * 1.02) + 3; }

/* what a tile's cells are and what is wanted of them */
enum {
    OT_ENGINE = 0, /* quart cells; the first leaf in tree order at the minimum */
    OT_CHUNK = 1,  /* quart cells; the chunk-cell rule (cell_chunk) */
    OT_BLOCK = 2,  /* blocks `step` <= 4 apart, zoomed to quart cells; the chunk-cell rule */
    OT_CHAIN = 3   /* quart cells; ENGINE's leaf with its target, distance and tie flag for the candidate chains */
};

/* s = x f + off as the reference rounds it (f a power of two, |x f| < 2^23: the wrap is the identity), floor i and
 * fraction F in units of 2^-64, from the mantissa of s as a signed 64-bit integer (an arithmetic shift of the negated
 * mantissa floors): one FP64-pipe operation, of which an SM completes two lanes per clock.  False for |s| < 2^-11,
 * |s| >= 2^20 and s in (-1, 0), where the reference's difference s - floor(s) rounds. */
__device__ __forceinline__ bool ot_split(double x, double f, double off, int &i, uint64_t &F) {
    const double s = __fma_rn(x, f, off);
    const uint32_t h = (uint32_t)__double2hiint(s);
    const int e = (int)((h >> 20) & 0x7FFu) - 1023;
    const int64_t m = (int64_t)(((uint64_t)((h & 0xFFFFFu) | 0x100000u) << 32) | (uint32_t)__double2loint(s));
    const int64_t neg = (int64_t)((int32_t)h >> 31);
    const int64_t M = (m ^ neg) - neg; /* s in units of 2^(e - 52) */
    i = (int32_t)(M >> 32) >> (20 - e);
    F = (uint64_t)M << (12 + e);
    return (uint32_t)(e + 11) <= 30u && (e >= 0 || (int32_t)h >= 0);
}
/* the rest, out of line; the product is volatile so that the compiler does not compute it ahead of the branch */
static __device__ __noinline__ SplitF ot_split_f_slow(double x, double f, double off) {
    SplitF r;
    double v;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(v) : "d"(x), "d"(f));
    split_f_plain(v, off, r.i, r.f);
    return r;
}
/* the float branch's split.  The hardware's u64 -> f32 conversion runs at the FP64 pipe's rate (595 Gop/s; u32 -> f32
 * 18,700), so the fraction is converted from its upper 32 bits (below 2^-7: its next 32) with the lower ones as a sticky
 * bit: 26 or more significant bits, whose guard and sticky bits round as the whole fraction does.  Fractions below 2^-14
 * take the plain path. */
__device__ __forceinline__ void ot_split_f(double x, double f, double off, int &i, float &fr) {
    uint64_t F;
    const bool ok = ot_split(x, f, off, i, F);
    uint32_t hi = (uint32_t)(F >> 32), lo = (uint32_t)F;
    float sc = 0x1.0p-32f;
    if (hi < (1u << 25)) {
        hi = __funnelshift_l(lo, hi, 7);
        lo <<= 7;
        sc = 0x1.0p-39f;
    }
    fr = __uint2float_rn(hi | (lo ? 1u : 0u)) * sc;
    if (!ok || hi < (1u << 25)) {
        const SplitF r = ot_split_f_slow(x, f, off);
        i = r.i;
        fr = r.f;
    }
}

/* where the nodes of one octave lie: first node (ib, kb) of the plane, nodes per row, place in the table */
struct OtRange {
    int32_t ib, kb, nx, off;
};
/* one octave in evaluation order (a noise's levels, first then second stack of each) */
struct __align__(16) OtOctF {
    double ox, oz; /* x and z offsets */
    double f;      /* input factor */
    float amp;     /* layer amplitude */
    float uy;      /* smoothstep of the zero coordinate's fraction */
    OtRange r;
};
/* entry of the shift tables: fraction, fraction - 1, smoothstep, node index part */
struct __align__(16) OtShiftF {
    float f, g, u;
    int32_t node;
};

/* work units of a table build: table t's nodes in units of 32, unit0[t] its first unit (non-decreasing) */
struct OtBuild {
    int32_t unit0[64];
    int16_t n[64], nx[64];
    int32_t inv[64]; /* ceil(65536 / nx): row = node * inv >> 16 for node < 1024, nx <= 32 */
    int32_t units;
};
/* the table that unit u belongs to (all lanes call it) */
__device__ __forceinline__ int ot_find_unit(const OtBuild &b, int u) {
    const int l = threadIdx.x & 31;
    return __popc(__ballot_sync(0xFFFFFFFFu, b.unit0[l] <= u)) + __popc(__ballot_sync(0xFFFFFFFFu, b.unit0[l + 32] <= u)) - 1;
}

/* one octave of the float branch from its four nodes (octave_q<float>'s operations on the same values: a node's
 * gradient dot is fma(g2, y, fma(g1, x, c)) with c the fixed coordinate's exact product; two of the three
 * components are non-zero, so one operation rounds, whatever the order).  Input (x, 0, z) (Z0 false): the node's two
 * gradients are those of the planes y and y + 1, t the fixed smoothstep of y; input (x, y, 0) (Z0 true): those of z and
 * z + 1, t that of z, and (a, b) = (x, y). */
struct OtNodeF {
    float4 p; /* g1, g2, c of the lower plane; g1 of the upper */
    float2 q; /* g2, c of the upper plane */
};
__device__ __forceinline__ float ot_dot0(const OtNodeF &n, float a, float b) { return __fmaf_rn(n.p.y, b, __fmaf_rn(n.p.x, a, n.p.z)); }
__device__ __forceinline__ float ot_dot1(const OtNodeF &n, float a, float b) { return __fmaf_rn(n.q.x, b, __fmaf_rn(n.p.w, a, n.q.y)); }
template <bool Z0>
__device__ __forceinline__ float ot_octave_f(const float4 *__restrict__ P, const float2 *__restrict__ Q, int at, int nx, float a,
                                             float ga, float u, float b, float gb, float v, float t) {
    const OtNodeF n00{P[at], Q[at]}, n10{P[at + 1], Q[at + 1]}, n01{P[at + nx], Q[at + nx]}, n11{P[at + nx + 1], Q[at + nx + 1]};
    const float l0 = lerp<float>(u, ot_dot0(n00, a, b), ot_dot0(n10, ga, b));   /* lower plane, row k */
    const float l1 = lerp<float>(u, ot_dot0(n01, a, gb), ot_dot0(n11, ga, gb)); /* lower plane, row k + 1 */
    const float h0 = lerp<float>(u, ot_dot1(n00, a, b), ot_dot1(n10, ga, b));
    const float h1 = lerp<float>(u, ot_dot1(n01, a, gb), ot_dot1(n11, ga, gb));
    /* the reference lerps x, then y, then z */
    if (Z0) return lerp<float>(t, lerp<float>(v, l0, l1), lerp<float>(v, h0, h1));
    return lerp<float>(v, lerp<float>(t, l0, h0), lerp<float>(t, l1, h1));
}

/* node (i, k) of lattice L: the gradients of its two planes, as the octave above reads them */
__device__ __forceinline__ void ot_node_f(const MgLattice &L, bool z0, int i, int k, float4 &p, float2 &q) {
    const PlainPerm P{L.p};
    const int a = P(i);
    float4 g0, g1;
    float c0, c1;
    if (z0) { /* (i, k) = (x, y) */
        const int aa = P(a + k);
        g0 = __ldg(&kGradF[P(aa + L.iz) & 15]);
        g1 = __ldg(&kGradF[P(aa + L.iz + 1) & 15]);
        c0 = g0.z * L.z0.f.fz;
        c1 = g1.z * (L.z0.f.fz - 1.0f);
        p = make_float4(g0.x, g0.y, c0, g1.x);
        q = make_float2(g1.y, c1);
    } else { /* (i, k) = (x, z) */
        g0 = __ldg(&kGradF[P(P(a + L.iy) + k) & 15]);
        g1 = __ldg(&kGradF[P(P(a + L.iy + 1) + k) & 15]);
        c0 = g0.y * L.z0.f.fy;
        c1 = g1.y * (L.z0.f.fy - 1.0f);
        p = make_float4(g0.x, g0.z, c0, g1.x);
        q = make_float2(g1.z, c1);
    }
}

/* ============================================================================ double branch
 * The double branch's five climate noises and ridges_folded reach the biome only through quantised targets (steps of 1e-4),
 * so the tile form evaluates them in 32-bit fixed point with 64-bit accumulators (no FP64 pipe, which the exact shift octaves
 * of the per-cell form kept 55 % busy) and takes a target when every value within the form's error bound has it
 * (MgNoise::tile_eq).  About 2 % of the cells keep a target open between two values; nearly all of them have the same biome for
 * both, and the rest (0.1 %) go to the exact evaluation of a later launch.
 *
 * Over a plane of the lattice an octave is V = (1 - W) L0 + W L1 with a row's value L = P + U Q, P = N0 and Q = N1 - N0
 * linear in the fractions (X, Z): N = A dx + B dz + C, whose A, B and C mix the two planes' gradients by the fixed
 * coordinate's smoothstep v: A = (1 - v) g0.x + v g1.x.  (The reference lerps x, then y, then z; the order only matters for
 * its roundings.)  The table holds one edge per pair of nodes (i, k), (i + 1, k): P's and Q's coefficients. */
struct OtEdge {
    int4 p; /* P: X and Z coefficients (units of 2^-29), constant (2^-28); Q: X coefficient (2^-30) */
    int2 q; /* Q: Z coefficient (2^-30), constant (2^-29) */
};
/* the fixed coordinate's part of an octave's edges, in units of 2^-30: v, 1 - v, Y (1 - v), (Y - 1) v */
struct __align__(16) OtFix {
    int32_t v, w, c0, c1;
};
__device__ __forceinline__ OtFix ot_fix(double y, double v) {
    OtFix f;
    f.v = __double2int_rn(v * 0x1.0p30);
    f.w = (1 << 30) - f.v;
    f.c0 = __double2int_rn(y * (1.0 - v) * 0x1.0p30);
    f.c1 = __double2int_rn((y - 1.0) * v * 0x1.0p30);
    return f;
}
/* entry of the shift tables: fraction and smoothstep (units of 2^-31), edge index part */
struct __align__(16) OtShiftD {
    int32_t f, u, edge, pad;
};
/* one climate octave in evaluation order; offsets in units of 2^-32, less the first node's cell */
struct __align__(16) OtOctD {
    int64_t ox, oz;
    int32_t nx, off; /* edges per row, place in the table */
    int32_t k, c30;  /* input factor 2^-k; level constant */
};
__device__ __forceinline__ int64_t ot_madw(int32_t a, int32_t b, int64_t c) {
    int64_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
__device__ __forceinline__ int32_t ot_hi(int64_t v) { return (int32_t)(v >> 32); }
__device__ __forceinline__ int32_t ot_sub_sat(int32_t a, int32_t b) {
    int32_t r;
    asm("sub.sat.s32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
#define OT_STACK_C ((int64_t)((MG_SECOND_STACK - 1.0) * 0x1.0p64)) /* exact */
/* smoothstep of the fraction t (units of 2^-32) in units of 2^-31: t > 1/2 as 1 - smoothstep(1 - t), and with t' = 2 t <= 1,
 * t^3 (10 - 15 t + 6 t^2) = t'^3 / 8 (10 - t' (7.5 - 1.5 t')).  The 2 centres the truncations: within 1.43e-9 (all 2^32
 * fractions evaluated). */
__device__ __forceinline__ int32_t ot_fade31(uint32_t t) {
    const int32_t m = (int32_t)t >> 31;
    const uint32_t tt = (t ^ (uint32_t)m) << 1;
    const uint32_t t3 = __umulhi(__umulhi(tt, tt), tt);
    const uint32_t p = (10u << 28) - __umulhi(tt, 15u * (1u << 27) - 2u - (tt >> 5) * 3u);
    return (int32_t)__umulhi(t3, p) ^ (m & 0x7FFFFFFF);
}
/* a row's value in units of 2^-60 from its edge; X and dz in units of 2^-31, dz in [-1, 1] */
__device__ __forceinline__ int64_t ot_row_d(const OtEdge &e, int32_t X, int32_t dz, int32_t U) {
    const int64_t q = ot_madw(e.p.w, X, ot_madw(e.q.x, dz, (int64_t)(((uint64_t)(uint32_t)e.q.y << 32) | 0x80000000u)));
    return ot_madw(U, ot_hi(q), ot_madw(e.p.x, X, ot_madw(e.p.y, dz, (int64_t)((uint64_t)(uint32_t)e.p.z << 32))));
}
/* the octave in units of 2^-60; X, Z, U, W in units of 2^-31 */
__device__ __forceinline__ int64_t ot_octave_d(const int4 *__restrict__ P, const int2 *__restrict__ Q, int at, int nx, int32_t X,
                                               int32_t U, int32_t Z, int32_t W) {
    const int64_t l0 = ot_row_d(OtEdge{P[at], Q[at]}, X, Z, U);
    const int64_t l1 = ot_row_d(OtEdge{P[at + nx], Q[at + nx]}, X, (int32_t)((uint32_t)Z - 0x80000000u), U);
    return ot_madw(W, ot_hi((int64_t)((uint64_t)(l1 - l0) << 1)), l0);
}
/* node (i, k) of lattice L in units of 2^-30: (A, B, C) */
__device__ __forceinline__ void ot_mix(int h0, int h1, bool z0, const OtFix &f, int32_t &A, int32_t &B, int32_t &C) {
    const int4 g = __ldg(&kGradI[h0 & 15]), h = __ldg(&kGradI[h1 & 15]);
    A = g.x * f.w + h.x * f.v;
    B = z0 ? g.y * f.w + h.y * f.v : g.z * f.w + h.z * f.v;
    C = z0 ? g.z * f.c0 + h.z * f.c1 : g.y * f.c0 + h.y * f.c1;
}
/* edge (i, k) - (i + 1, k) of the plane at `fixed` (the cell of the fixed coordinate) */
template <typename PERM>
__device__ __forceinline__ void ot_edge(const PERM &P, int fixed, bool z0, const OtFix &f, int i, int k, int4 &p, int2 &q) {
    const int a = P(i), b = P(i + 1);
    int h0, h1, h2, h3;
    if (z0) {
        const int aa = P(a + k) + fixed, bb = P(b + k) + fixed;
        h0 = P(aa); h1 = P(aa + 1); h2 = P(bb); h3 = P(bb + 1);
    } else {
        h0 = P(P(a + fixed) + k); h1 = P(P(a + fixed + 1) + k); h2 = P(P(b + fixed) + k); h3 = P(P(b + fixed + 1) + k);
    }
    int32_t A0, B0, C0, A1, B1, C1;
    ot_mix(h0, h1, z0, f, A0, B0, C0);
    ot_mix(h2, h3, z0, f, A1, B1, C1);
    p = make_int4((A0 + 1) >> 1, (B0 + 1) >> 1, (C0 + 2) >> 2, ot_sub_sat(A1, A0));
    q = make_int2(ot_sub_sat(B1, B0), (int32_t)(((int64_t)C1 - A1 - C0 + 1) >> 1));
}
__device__ __forceinline__ void ot_edge(const MgLattice &L, bool z0, const OtFix &f, int i, int k, int4 &p, int2 &q) {
    ot_edge(PlainPerm{L.p}, z0 ? L.iz : L.iy, z0, f, i, k, p, q);
}
/* ot_octave_d for one sample of a lattice, its two edges built on the way */
template <typename PERM>
__device__ __forceinline__ int64_t ot_sample_d(const PERM &P, int fixed, bool z0, const OtFix &f, int i, int k, int32_t X, int32_t U,
                                               int32_t Z, int32_t W) {
    OtEdge e0, e1;
    ot_edge(P, fixed, z0, f, i, k, e0.p, e0.q);
    ot_edge(P, fixed, z0, f, i, k + 1, e1.p, e1.q);
    const int64_t l0 = ot_row_d(e0, X, Z, U), l1 = ot_row_d(e1, X, (int32_t)((uint32_t)Z - 0x80000000u), U);
    return ot_madw(W, ot_hi((int64_t)((uint64_t)(l1 - l0) << 1)), l0);
}
/* cell, fraction and smoothstep (units of 2^-31, as the shift tables hold them) of a whole coordinate c (or its second-stack
 * multiple) times f plus off */
__device__ __forceinline__ void ot_split_d(double c, double f, double off, int &i, int32_t &t, int32_t &u) {
    uint64_t F;
    if (!ot_split(c, f, off, i, F)) { /* rare: the sum near zero or beyond 2^20 */
        const double s = __fma_rn(c, f, off);
        i = ifloor(s);
        F = (uint64_t)__double2ll_rn((s - (double)i) * 0x1.0p63) << 1;
    }
    t = (int32_t)min((uint32_t)(((F >> 32) + 1) >> 1), 0x7FFFFFFFu);
    u = (int32_t)min((uint32_t)((fadeq((int64_t)(F >> (64 - MG_Q))) + (1LL << 27)) >> 28), 0x7FFFFFFFu);
}
/* the targets a value within e of v may have (units of 2^-29, 2^-28 for the depth: `scale` is 10000 times the unit): the
 * rounding to float, the product by 10000 and the truncation are each monotone, so the ends' targets bound it */
__device__ __forceinline__ void ot_target(int32_t v, int32_t e, float scale, int32_t &a, int32_t &b) {
    a = __float2int_rz(__int2float_rn(v - e) * scale);
    b = __float2int_rz(__int2float_rn(v + e) * scale);
}

/* The offset spline with a bound: at coordinates within de of the reference's, the value is within `err` of the reference's.
 * A coordinate within de of an end of its segment may lie in the neighbouring one for the reference, whose roundings and curvature
 * are others: the cell is left open (coordinates are within 4e-7, so that this is a few cells in 10^5).  Else both evaluate the
 * same segment: its value is a convex combination of its two points' values (so their errors pass through at most) plus a cubic in
 * t, whose slope in the input is at most (|y2 - y1| + 1.25 (|a| + |b|)) / (x2 - x1), 3.5 (e1 + e2) / (x2 - x1) more where the
 * points' values are within e1 and e2; the roundings of one evaluation are within 2^-24 times 2 u_t = 2 (|y2 - y1| +
 * 1.25 (|a| + |b|)) for t's two, 2 |y2 - y1| + max |y| for the first lerp, a quarter of |y2 - y1| and 1.75 (|a| + |b|) for the
 * cubic, max |y| + 0.25 (|a| + |b|) for the sum: 4.25 |y2 - y1| + 2 max |y| + 4.5 (|a| + |b|), and both sides round.  A constant
 * segment has no roundings. */
#define OT_SPL_DEPTH 4 /* nesting levels unrolled (every 26.x table: 4) */
struct SplineIn {
    float c, e, r, f;     /* continents, erosion, ridges, ridges_folded */
    float dc, de, dr, df; /* their bounds */
};
/* the value below reference c.  One copy of the code per nesting level, its state in registers: an explicit stack keeps it in
 * local memory, and measured three times slower here. */
template <int D>
__device__ __forceinline__ float spline_err(const MgSpline &S, int c, const SplineIn &x, float &err) {
    err = 0.0f;
    if (c < 0) return S.cval[~c];
    if constexpr (D == 0) {
        err = 1e30f; /* nested deeper: the cell is left open */
        return 0.0f;
    } else {
        const int o = S.first[c], n = S.npts[c], k = S.coord[c];
        const float in = k == 0 ? x.c : (k == 1 ? x.e : (k == 2 ? x.r : x.f));
        const float de = k == 0 ? x.dc : (k == 1 ? x.de : (k == 2 ? x.dr : x.df));
        int i = -1; /* last point at or below the input */
        for (int j = 0; j < n; j++) i += in >= S.loc[o + j] ? 1 : 0;
        const bool ext = i < 0 || i == n - 1;
        const int p = o + max(i, 0);
        float y1 = 0.0f, e1 = 0.0f, y2 = 0.0f, e2 = 0.0f;
#pragma unroll 1
        for (int q = 0; q < (ext ? 1 : 2); q++) {
            y1 = y2;
            e1 = e2;
            y2 = spline_err<D - 1>(S, S.child[p + q], x, e2);
        }
        const float x1 = S.loc[p], d1 = S.der[p], dx = in - x1;
        if (ext) { /* linear extension */
            const float v = d1 * dx;
            err = d1 == 0.0f ? e2 : e2 + fabsf(d1) * 1.001f * de + 1.2e-7f * (4.0f * fabsf(v) + fabsf(y2));
            if (fabsf(dx) <= 1.001f * de) err = 1e30f;
            return d1 == 0.0f ? y2 : y2 + v;
        }
        const float x2 = S.loc[p + 1], w = x2 - x1, t = dx / w, d2 = S.der[p + 1], dy = y2 - y1;
        const float a = d1 * w - dy, b = -d2 * w + dy;
        const float ab = fabsf(a) + fabsf(b), ad = fabsf(dy);
        err = fmaxf(e1, e2) + __fdividef(ad + 1.25f * ab + 3.5f * (e1 + e2), w) * 1.001f * de +
              1.2e-7f * (4.3f * ad + 2.0f * fmaxf(fabsf(y1), fabsf(y2)) + 4.6f * ab);
        if (ad + ab + e1 + e2 == 0.0f) err = 0.0f;
        if (fminf(dx, x2 - in) <= 1.001f * de) err = 1e30f;
        return lerp<float>(t, y1, y2) + t * (1.0f - t) * lerp<float>(t, a, b);
    }
}

/* targets [ta, tb] of the five climate noises' values v (units of 2^-29, v[q - 1] within eq[q] of noise q's) and the depth
 * gradient plus offset (units of 2^-28); es: the offset spline's error bound, 1 or more when the targets do not hold */
__device__ __forceinline__ void ot_climate_targets(const MgWorldDesc &W, const MgSpline &S, const int32_t (&v)[MG_OW_NOISES - 1],
                                                   const int32_t (&eq)[MG_OW_NOISES], int32_t depth, int32_t (&ta)[6], int32_t (&tb)[6],
                                                   float &es) {
    const float s29 = 10000.0f * 0x1.0p-29f, s28 = 10000.0f * 0x1.0p-28f;
    const int32_t ec = eq[3], ee = eq[4], ew = eq[5];
    ot_target(v[0], eq[1], s29, ta[0], tb[0]);
    ot_target(v[1], eq[2], s29, ta[1], tb[1]);
    ot_target(v[2], ec, s29, ta[2], tb[2]);
    ot_target(v[3], ee, s29, ta[3], tb[3]);
    ot_target(v[4], ew, s29, ta[5], tb[5]);
    /* spline coordinates: floats of the values, of ridges_folded (|(|r| + c0)| + c1) c2 (the sums in units of
     * 2^-29); each within its noise's bound (times |c2|) and both sides' roundings to float */
    const float u = 0x1.0p-29f;
    const int32_t rs = abs(abs(v[4]) + (int32_t)((W.rf_q[0] + (1 << 29)) >> 30)) + (int32_t)((W.rf_q[1] + (1 << 29)) >> 30);
    const float c2 = (float)W.rf_d[2] * u;
    SplineIn si;
    si.c = (float)v[2] * u;
    si.e = (float)v[3] * u;
    si.r = (float)v[4] * u;
    si.f = (float)rs * c2;
    si.dc = (float)ec * u + fabsf(si.c) * 1.2e-7f;
    si.de = (float)ee * u + fabsf(si.e) * 1.2e-7f;
    si.dr = (float)ew * u + fabsf(si.r) * 1.2e-7f;
    si.df = fabsf(c2) * (float)(ew + 2) + fabsf(si.f) * 1.9e-7f;
    float sp = spline_err<OT_SPL_DEPTH>(S, S.root, si, es);
    if (fabsf(sp) > 3.9f) { /* the depth (|gradient + offset| < 3: ow_tile_supported) must fit its units: left open */
        sp = 0.0f;
        es = 1e30f;
    }
    ot_target(depth + __float2int_rn(sp * 0x1.0p28f), (int32_t)(es * (1.01f * 0x1.0p28f)) + 3, s28, ta[4], tb[4]);
}

/* ---- one cell of its own (neighbours that share no tables): its octaves' edges are built on the way */
/* the lattices' fixed coordinates' parts (fz: of the shift's z planes) and offsets in units of 2^-32, by threads t of nt */
__device__ __forceinline__ void ot_cell_fix(const MgWorldDesc &W, const MgLattice *lat, OtFix *fix, OtFix *fz, int64_t (*off)[2], int t,
                                            int nt) {
    for (int l = t; l < W.ntables; l += nt) {
        const MgLattice &L = lat[l];
        fix[l] = ot_fix(L.fyd, L.uyd);
        if (l < 2 * W.noise[0].nlev) fz[l] = ot_fix(L.fzd, L.uzd);
        off[l][0] = __double2ll_rn(L.ox * 0x1.0p32);
        off[l][1] = __double2ll_rn(L.oz * 0x1.0p32);
    }
}
/* the five climate noises of quart cell (cx, cz), |cx|, |cz| < OT_COORD_LIM: values v in units of 2^-29, v[n - 1] within eq[n] of
 * noise n's */
__device__ __forceinline__ void ot_cell_d(const MgWorldDesc &W, const MgLattice *lat, const OtFix *fix, const OtFix *fz,
                                          const int64_t (*off)[2], int cx, int cz, int32_t (&v)[MG_OW_NOISES - 1],
                                          int32_t (&eq)[MG_OW_NOISES]) {
    const MgNoise &O = W.noise[0];
    int64_t sa = 0, sb = 0; /* units of 2^-59 */
#pragma unroll 1
    for (int k = 0; k < O.nlev; k++) {
        int64_t va = 0, vb = 0;
#pragma unroll 1
        for (int st = 0; st < 2; st++) {
            const int l = st * O.nlev + k;
            const MgLattice &L = lat[l];
            const PlainPerm P{L.p};
            double X = (double)cx, Z = (double)cz;
            if (st) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
            int ia, ib;
            int32_t pa, ua, pb, ub;
            ot_split_d(X, O.freq[k], L.ox, ia, pa, ua);
            ot_split_d(Z, O.freq[k], L.oz, ib, pb, ub);
            va += ot_sample_d(P, L.iy, false, fix[l], ia, ib, pa, ua, pb, ub);
            ot_split_d(Z, O.freq[k], L.ox, ia, pa, ua);
            ot_split_d(X, O.freq[k], L.oy, ib, pb, ub);
            vb += ot_sample_d(P, L.iz, true, fz[l], ia, ib, pa, ua, pb, ub);
        }
        sa = ot_madw((int32_t)(va >> 31), O.c30[k], sa);
        sb = ot_madw((int32_t)(vb >> 31), O.c30[k], sb);
    }
    const int64_t x = ((int64_t)cx << 32) + (sa >> 25), z = ((int64_t)cz << 32) + (sb >> 25);
    const int64_t xc = x + __mul64hi(x, OT_STACK_C), zc = z + __mul64hi(z, OT_STACK_C);
    const bool out17 = max(abs(cx), abs(cz)) >= (1 << 17) - OT_W;
#pragma unroll 1
    for (int n = 1; n < MG_OW_NOISES; n++) {
        const MgNoise &N = W.noise[n];
        int64_t acc = 0;
#pragma unroll 1
        for (int k = 0; k < N.nlev; k++) {
            int64_t lev = 0;
#pragma unroll 1
            for (int st = 0; st < 2; st++) {
                const int l = N.base + st * N.nlev + k;
                const MgLattice &L = lat[l];
                const int64_t sx = ((st ? xc : x) >> -N.fexp[k]) + off[l][0], sz = ((st ? zc : z) >> -N.fexp[k]) + off[l][1];
                lev += ot_sample_d(PlainPerm{L.p}, L.iy, false, fix[l], ot_hi(sx), ot_hi(sz), (int32_t)((uint32_t)sx >> 1),
                                   ot_fade31((uint32_t)sx), (int32_t)((uint32_t)sz >> 1), ot_fade31((uint32_t)sz));
            }
            acc = ot_madw((int32_t)(lev >> 31), N.c30[k], acc);
        }
        const int32_t e = out17 ? N.tile_eq_far : N.tile_eq;
#pragma unroll
        for (int k = 1; k < MG_OW_NOISES; k++) {
            v[k - 1] = n == k ? (int32_t)(acc >> 30) : v[k - 1];
            eq[k] = n == k ? e : eq[k];
        }
    }
}

}  // namespace mg
#endif
