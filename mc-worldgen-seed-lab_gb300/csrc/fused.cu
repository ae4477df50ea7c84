/* fused.cu -- many seeds x fixed points, Overworld: k_ow_seed_climate + k_ow_finish_tree.
 *
 * One CTA owns S seeds and one thread owns one lattice of one seed (46 per Overworld seed).  A thread
 * shuffles its permutation in shared memory (interleaved layout: byte i of thread t in word [i >> 2][t],
 * so all of a thread's accesses hit bank t % 32) and then samples *its own* lattice at every point of its
 * seed -- the lattices never leave the SM and their lookups never conflict.  Per-lattice octave values go
 * to shared memory, and one thread per (seed, point) sums them in the reference's order
 * (engine/mc_noise.h:285-324), forms the shifted coordinates after the ShiftA/ShiftB pass
 * (engine/mc_climate.h:113-164) and writes the five noise values.  k_ow_finish_tree then finishes the
 * climate with one thread per sample and searches the R-tree (ENGINE rule) for a warp's 32 samples one after another, 32
 * boxes at a time (tree_search_lanes: 957 -> 470 us for 65,536 seeds x 8 points), at full occupancy: inside the
 * fused kernel that serial per-point work would leave most of a CTA idle at its barriers.
 *
 * Phases per chunk of NPC points:  B  offset lattices: ShiftA and ShiftB octaves
 *                                   C  (seed, point): shift sums -> shifted x, z
 *                                   D  climate lattices: octaves at the shifted coordinates
 *                                   E  (seed, point): noise sums -> clim
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "batch.h"
#include "climate.cuh"
#include "launch.h"
#include "owtile.cuh"
#include "search.cuh"
#include "prof.h"

namespace mg {

/* threads per CTA: 4 seeds x 46 lattices, no idle thread, so that the float branch's shared memory (55.9 KB:
 * 64 permutation rows of FPS words, the chunk's octave values, offset headers) fits 4 CTAs per SM; the
 * double branch's (63.3 KB, values in double) fits 3 */
#define FNT 184
/* words per permutation row: byte i of thread t's permutation is in word [i >> 2][t]; a row of a multiple of
 * 32 words puts every thread's bytes in bank t % 32 whatever the row, so the shuffle's random swaps never
 * conflict (with 184 words a swap's bank would depend on its row) */
#define FPS 192
#define FNPC 8  /* points per chunk */
#define FMAXT 48 /* lattices per seed this kernel supports */

#define FMAXS 4  /* seeds per CTA at 46 lattices per seed */
#define FMAXOFF 24 /* offset-noise lattices per CTA (6 per seed) */

/* header of an offset-noise lattice, shared so that any thread can sample it: all of it for the double
 * branch, the fields the float branch's octaves read (offsets, floors, zero-coordinate split) for the float */
struct OffHdr {
    double ox, oy, oz, fyd, fzd, uyd, uzd;
    int64_t Fy, Fz;
    int iy, iz;
    MgLatZero z0;
};
struct OffHdrF {
    double ox, oy, oz;
    int iy, iz;
    MgLatZero z0;
    __device__ OffHdrF &operator=(const OffHdr &h) {
        ox = h.ox; oy = h.oy; oz = h.oz; iy = h.iy; iz = h.iz; z0 = h.z0;
        return *this;
    }
};

template <typename V>
struct FusedSmem {
    uint32_t perm[64][FPS];
    V val[FNT][FNPC];               /* octave value of lattice (owner thread) t at point p of the chunk */
    union {                         /* valb until phase C has read it, then coord (phase C syncs between) */
        V valb[FMAXOFF][FNPC];      /* ShiftB octave of the offset lattices */
        double coord[FMAXS][FNPC][4]; /* per (seed, point): x, z, x*c, z*c */
    };
    typename std::conditional<std::is_same<V, float>::value, OffHdrF, OffHdr>::type hdr[FMAXOFF];
};

/* lattice j of a seed (engine/mc_climate.h:95-106, engine/mc_noise.h:29-41), its permutation into a column of FusedSmem::perm */
struct FusedOwn {
    int noise = 0, st = 0, lev = 0;
    double ox = 0.0, oy = 0.0, oz = 0.0;
};
__device__ __forceinline__ void fused_lattice(const MgWorldDesc &W, int64_t seed, int j, uint32_t *col, FusedOwn &o) {
    while (o.noise < MG_OW_NOISES - 1 && j >= W.noise[o.noise + 1].base) o.noise++;
    const MgNoise &N = W.noise[o.noise];
    const int r = j - N.base;
    o.st = r >= N.nlev;
    o.lev = r - o.st * N.nlev;
    Xo root = xo_from_seed(seed);
    uint64_t plo = xo_next(root), phi = xo_next(root);
    Xo nr = xo_make(W.nhl[o.noise] ^ plo, W.nhh[o.noise] ^ phi);
    uint64_t a = xo_next(nr), b = xo_next(nr);
    if (o.st) { a = xo_next(nr); b = xo_next(nr); }
    Xo x = xo_make(N.hlo[o.lev] ^ a, N.hhi[o.lev] ^ b);
    o.ox = xo_double(x) * 256.0;
    o.oy = xo_double(x) * 256.0;
    o.oz = xo_double(x) * 256.0;
    for (int w = 0; w < 64; w++) col[w * FPS] = 0x03020100u + 0x04040404u * (uint32_t)w;
    xo_shuffle<FPS>(reinterpret_cast<uint8_t *>(col), x); /* byte i at col + (i >> 2) * 4 FPS + (i & 3) */
}

/* Threads are lattice-major: thread t owns lattice j = t / spc of local seed t % spc, so the offset-noise
 * lattices of all the CTA's seeds are threads 0 .. noff*spc-1 and their shift octaves (16 per point) can be
 * spread over every thread of the CTA in phase B. */
template <bool FM>
__global__ void __launch_bounds__(FNT) k_ow_seed_climate(const __grid_constant__ MgWorldDesc W,
                                                         const int64_t *__restrict__ seeds, int ns,
                                                         const int32_t *__restrict__ pts, int np,
                                                         typename std::conditional<FM, float, double>::type *__restrict__ clim) {
    typedef typename std::conditional<FM, float, double>::type V;
    extern __shared__ uint4 smem_raw[];
    FusedSmem<V> &sm = *reinterpret_cast<FusedSmem<V> *>(smem_raw);
    const int t = threadIdx.x;
    const int nt = W.ntables;
    const int spc = FNT / nt;                 /* seeds per CTA */
    const int s0 = blockIdx.x * spc;          /* first seed of the CTA */
    const int j = t / spc, ls = t % spc;      /* lattice index, local seed */
    const bool active = j < nt && s0 + ls < ns;
    const MgNoise &O = W.noise[0];
    const int noff = 2 * O.nlev;              /* offset-noise lattices per seed (noise 0 is first) */
    const int nown = noff * spc;              /* offset-noise lattice owners in the CTA */

    /* ---- phase A: this thread's lattice */
    FusedOwn own;
    if (active) fused_lattice(W, seeds[s0 + ls], j, &sm.perm[0][t], own);
    const int noise = own.noise, st = own.st, lev = own.lev;
    const double ox = own.ox, oy = own.oy, oz = own.oz;
    /* split of the offsets used by a zero input coordinate */
    OffHdr h;
    h.ox = ox; h.oy = oy; h.oz = oz;
    lattice_header(h, !FM);
    if (t < nown) sm.hdr[t] = h;
    const uint8_t *pbase = reinterpret_cast<const uint8_t *>(&sm.perm[0][0]);
    const MgNoise &N = W.noise[noise];
    const double f = N.freq[lev];
    const int fk = N.fexp[lev];

    for (int p0 = 0; p0 < np; p0 += FNPC) {
        const int npc = min(FNPC, np - p0);
        __syncthreads(); /* lattices and headers complete / previous chunk consumed */
        /* ---- phase B: ShiftA (x, 0, z) and ShiftB (z, x, 0) octaves, item = (owner, point) */
        for (int item = t; item < nown * npc; item += FNT) {
            const int o = item % nown, p = item / nown;
            const int oj = o / spc;
            const int ost = oj >= O.nlev, olev = oj - ost * O.nlev;
            if (s0 + o % spc >= ns) continue;
            const auto &oh = sm.hdr[o];
            const IlvPerm<FPS> perm{pbase, o};
            const int32_t *pp = pts + 3 * (p0 + p);
            double X = (double)pp[0], Z = (double)pp[2];
            if (ost) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
            const double of = O.freq[olev];
            const int ok = O.fexp[olev];
            if constexpr (FM) {
                int ix, izz, iyy;
                float fx, fzz, fyy;
                split_fk(X, of, ok, oh.ox, ix, fx);
                split_fk(Z, of, ok, oh.oz, izz, fzz);
                sm.val[o][p] = (V)octave_y0<float>(perm, oh, ix, fx, izz, fzz);
                split_fk(Z, of, ok, oh.ox, ix, fx);
                split_fk(X, of, ok, oh.oy, iyy, fyy);
                sm.valb[o][p] = (V)octave_z0<float>(perm, oh, ix, fx, iyy, fyy);
            } else {
                int ix, izz, iyy;
                double fx, fzz, fyy;
                int64_t FX, FZ, FY;
                split_dk(X, of, ok, oh.ox, ix, fx, FX);
                split_dk(Z, of, ok, oh.oz, izz, fzz, FZ);
                sm.val[o][p] = (V)octave_d_y0(perm, oh, ix, fx, FX, izz, fzz, FZ);
                split_dk(Z, of, ok, oh.ox, ix, fx, FX);
                split_dk(X, of, ok, oh.oy, iyy, fyy, FY);
                sm.valb[o][p] = (V)octave_d_z0(perm, oh, ix, fx, FX, iyy, fyy, FY);
            }
        }
        __syncthreads();
        /* ---- phase C: shift sums and shifted coordinates, one thread per (seed, point) */
        double cx = 0.0, cz = 0.0;
        bool cw = false;
        if (t < spc * FNPC) {
            const int cs = t / FNPC, p = t % FNPC;
            if (p < npc && s0 + cs < ns) {
                const int32_t *pp = pts + 3 * (p0 + p);
                const double X = (double)pp[0], Z = (double)pp[2];
                double x, z;
                if (FM) {
                    float sa = 0.0f, sb = 0.0f;
                    for (int k = 0; k < O.nlev; k++) {
                        sa += O.amp_f[k] * (float)sm.val[k * spc + cs][p];
                        sa += O.amp_f[k] * (float)sm.val[(O.nlev + k) * spc + cs][p];
                    }
                    for (int k = 0; k < O.nlev; k++) {
                        sb += O.amp_f[k] * (float)sm.valb[k * spc + cs][p];
                        sb += O.amp_f[k] * (float)sm.valb[(O.nlev + k) * spc + cs][p];
                    }
                    x = X + (double)(sa * 4.0f);
                    z = Z + (double)(sb * 4.0f);
                } else {
                    double a1 = 0.0, a2 = 0.0, b1 = 0.0, b2 = 0.0;
                    for (int k = 0; k < O.nlev; k++) a1 += O.amp_d[k] * (double)sm.val[k * spc + cs][p] * O.vf_d[k];
                    for (int k = 0; k < O.nlev; k++) a2 += O.amp_d[k] * (double)sm.val[(O.nlev + k) * spc + cs][p] * O.vf_d[k];
                    for (int k = 0; k < O.nlev; k++) b1 += O.amp_d[k] * (double)sm.valb[k * spc + cs][p] * O.vf_d[k];
                    for (int k = 0; k < O.nlev; k++) b2 += O.amp_d[k] * (double)sm.valb[(O.nlev + k) * spc + cs][p] * O.vf_d[k];
                    x = X + ((a1 + a2) * O.vfac) * 4.0;
                    z = Z + ((b1 + b2) * O.vfac) * 4.0;
                }
                cx = x;
                cz = z;
                cw = true;
            }
        }
        __syncthreads(); /* every valb read is done: coord may overwrite it */
        if (cw) {
            const int cs = t / FNPC, p = t % FNPC;
            sm.coord[cs][p][0] = cx;
            sm.coord[cs][p][1] = cz;
            sm.coord[cs][p][2] = cx * MG_SECOND_STACK;
            sm.coord[cs][p][3] = cz * MG_SECOND_STACK;
        }
        __syncthreads();
        /* ---- phase D: climate octaves at (x, 0, z), each thread on its own lattice */
        if (active && noise != 0) {
            const IlvPerm<FPS> perm{pbase, t};
            for (int p = 0; p < npc; p++) {
                const double x = sm.coord[ls][p][st ? 2 : 0], z = sm.coord[ls][p][st ? 3 : 1];
                if (FM) {
                    int ix, izz;
                    float fx, fzz;
                    split_fk(x, f, fk, ox, ix, fx);
                    split_fk(z, f, fk, oz, izz, fzz);
                    sm.val[t][p] = (V)octave_y0<float>(perm, h, ix, fx, izz, fzz);
                } else {
                    int ix, izz;
                    double fx, fzz;
                    int64_t FX, FZ;
                    split_dk(x, f, fk, ox, ix, fx, FX);
                    split_dk(z, f, fk, oz, izz, fzz, FZ);
                    sm.val[t][p] = (V)octave_d_y0(perm, h, ix, fx, FX, izz, fzz, FZ);
                }
            }
        }
        __syncthreads();
        /* ---- phase E: the five noise sums of every (seed, point) -> clim[(s * np + p) * 5 + q] */
        if (t < spc * FNPC) {
            const int cs = t / FNPC, p = t % FNPC;
            if (p < npc && s0 + cs < ns) {
                V *dst = clim + ((size_t)(s0 + cs) * np + p0 + p) * 5;
                for (int q = 1; q < MG_OW_NOISES; q++) {
                    const MgNoise &Q = W.noise[q];
                    if (FM) {
                        float acc = 0.0f;
                        for (int k = 0; k < Q.nlev; k++) {
                            acc += Q.amp_f[k] * (float)sm.val[(Q.base + k) * spc + cs][p];
                            acc += Q.amp_f[k] * (float)sm.val[(Q.base + Q.nlev + k) * spc + cs][p];
                        }
                        dst[q - 1] = (V)acc;
                    } else {
                        double a1 = 0.0, a2 = 0.0;
                        for (int k = 0; k < Q.nlev; k++) a1 += Q.amp_d[k] * (double)sm.val[(Q.base + k) * spc + cs][p] * Q.vf_d[k];
                        for (int k = 0; k < Q.nlev; k++) a2 += Q.amp_d[k] * (double)sm.val[(Q.base + Q.nlev + k) * spc + cs][p] * Q.vf_d[k];
                        dst[q - 1] = (V)((a1 + a2) * Q.vfac);
                    }
                }
            }
        }
    }
}

/* a thread's octave at c = {x, z, and their second-stack multiples} */
template <bool FM, typename V>
__device__ __forceinline__ V search_octave(const MgWorldDesc &W, const FusedOwn &own, const OffHdr &h, const IlvPerm<FPS> &perm,
                                           const double *c) {
    const MgNoise &N = W.noise[own.noise];
    const double x = c[own.st ? 2 : 0], z = c[own.st ? 3 : 1], f = N.freq[own.lev];
    const int k = N.fexp[own.lev];
    int ix, iz;
    if constexpr (FM) {
        float fx, fz;
        split_fk(x, f, k, own.ox, ix, fx);
        split_fk(z, f, k, own.oz, iz, fz);
        return (V)octave_y0<float>(perm, h, ix, fx, iz, fz);
    } else {
        double fx, fz;
        int64_t FX, FZ;
        split_dk(x, f, k, own.ox, ix, fx, FX);
        split_dk(z, f, k, own.oz, iz, fz, FZ);
        return (V)octave_d_y0(perm, h, ix, fx, FX, iz, fz, FZ);
    }
}
/* a noise's sum of its octaves, in the reference's order (engine/mc_noise.h:285-324); first: val index of its first lattice */
template <bool FM, typename V>
__device__ __forceinline__ V search_sum(const MgNoise &N, const V *val, int first, int spc, int s) {
    if constexpr (FM) {
        float acc = 0.0f;
        for (int k = 0; k < N.nlev; k++) {
            acc += N.amp_f[k] * val[(first + k) * spc + s];
            acc += N.amp_f[k] * val[(first + N.nlev + k) * spc + s];
        }
        return acc;
    } else {
        double a1 = 0.0, a2 = 0.0;
        for (int k = 0; k < N.nlev; k++) a1 += N.amp_d[k] * val[(first + k) * spc + s] * N.vf_d[k];
        for (int k = 0; k < N.nlev; k++) a2 += N.amp_d[k] * val[(first + N.nlev + k) * spc + s] * N.vf_d[k];
        return (a1 + a2) * N.vfac;
    }
}

/* ---- the double branch's many seeds x points in the Overworld tiles' fixed point (owtile.cuh): the double evaluation's 72 FP64
 * operations an octave kept the FP64 pipe 73 % busy (1,501 seeds x 33 points: 383 us; this form 158, 221 with the queued samples
 * evaluated one at a time).  A sample whose targets the error bounds leave open (2 %) is kept in its seed's queue and evaluated in
 * double at the end, eight per seed at a time, from the lattices that are still there.  Writes the six targets of every sample. */
#define TQ_CAP 64 /* points whose values are kept until their targets are formed, by all threads at once */
struct TargetSmem {
    uint32_t perm[64][FPS];
    /* of the fixed point, and of the exact evaluation of the samples in the queues (FNPC of every seed at a time) */
    union {
        int64_t val[FNT][FNPC]; /* octave value of lattice (owner thread) t at point p of the chunk, units of 2^-60 */
        double val_d[FNT][FNPC];
    };
    union {
        int64_t sh[2][FMAXOFF][FNPC]; /* ShiftA, ShiftB octaves */
        double sh_d[2][FMAXOFF][FNPC];
    };
    union {
        int64_t coord[FMAXS][FNPC][4]; /* per (seed, point): x, z and their second-stack multiples, units of 2^-32 */
        double coord_d[FMAXS][FNPC][4];
    };
    struct {
        double ox, oy, oz;
        OtFix fy, fz;
        int iy, iz;
    } hdr[FMAXOFF];
    int32_t v[FMAXS][TQ_CAP][MG_OW_NOISES - 1]; /* units of 2^-29 */
    int queue[FMAXS][TQ_CAP], queued[FMAXS];
};
__global__ void __launch_bounds__(FNT, 3) k_ow_seed_targets(const __grid_constant__ MgWorldDesc W, const MgSpline *__restrict__ spline,
                                                            const int64_t *__restrict__ seeds, int ns, const int32_t *__restrict__ pts,
                                                            int np, int32_t *__restrict__ targets) {
    extern __shared__ uint4 smem_raw[];
    TargetSmem &sm = *reinterpret_cast<TargetSmem *>(smem_raw);
    const int t = threadIdx.x, nt = W.ntables, spc = FNT / nt, s0 = blockIdx.x * spc, j = t / spc, ls = t % spc;
    const bool active = j < nt && s0 + ls < ns;
    const MgNoise &O = W.noise[0];
    const int noff = 2 * O.nlev, nown = noff * spc;
    FusedOwn own;
    if (active) fused_lattice(W, seeds[s0 + ls], j, &sm.perm[0][t], own);
    OffHdr h;
    h.ox = own.ox; h.oy = own.oy; h.oz = own.oz;
    lattice_header(h, true);
    const OtFix fix = ot_fix(h.fyd, h.uyd);
    const int iy = h.iy, lev = -W.noise[own.noise].fexp[own.lev];
    const int64_t oxq = __double2ll_rn(own.ox * 0x1.0p32), ozq = __double2ll_rn(own.oz * 0x1.0p32);
    if (t < nown) {
        sm.hdr[t].ox = own.ox; sm.hdr[t].oy = own.oy; sm.hdr[t].oz = own.oz;
        sm.hdr[t].fy = fix;
        sm.hdr[t].fz = ot_fix(h.fzd, h.uzd);
        sm.hdr[t].iy = h.iy; sm.hdr[t].iz = h.iz;
    }
    if (t < FMAXS) sm.queued[t] = 0;
    const uint8_t *pbase = reinterpret_cast<const uint8_t *>(&sm.perm[0][0]);
    const IlvPerm<FPS> mine{pbase, t};

    /* the samples in the queues, FNPC of every seed at once, in double: k_ow_seed_climate's phases (all threads call it) */
    auto drain = [&]() {
        for (int r0 = 0;; r0 += FNPC) {
            __syncthreads();
            int most = 0;
            for (int s = 0; s < spc; s++) most = max(most, sm.queued[s]);
            if (r0 >= most) break;
            for (int item = t; item < nown * FNPC; item += FNT) {
                const int o = item % nown, r = item / nown, oj = o / spc, s = o % spc;
                if (r0 + r >= sm.queued[s]) continue;
                const IlvPerm<FPS> perm{pbase, o};
                const int32_t *pp = pts + 3 * sm.queue[s][r0 + r];
                OffHdr x;
                x.ox = sm.hdr[o].ox; x.oy = sm.hdr[o].oy; x.oz = sm.hdr[o].oz;
                lattice_header(x, true);
                const int lv = oj >= O.nlev ? oj - O.nlev : oj, k = O.fexp[lv];
                double X = (double)pp[0], Z = (double)pp[2];
                if (oj >= O.nlev) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
                const double f = O.freq[lv];
                int ix, iz, iyy;
                double fx, fz, fy;
                int64_t FX, FZ, FY;
                split_dk(X, f, k, x.ox, ix, fx, FX);
                split_dk(Z, f, k, x.oz, iz, fz, FZ);
                sm.sh_d[0][o][r] = octave_d_y0(perm, x, ix, fx, FX, iz, fz, FZ);
                split_dk(Z, f, k, x.ox, ix, fx, FX);
                split_dk(X, f, k, x.oy, iyy, fy, FY);
                sm.sh_d[1][o][r] = octave_d_z0(perm, x, ix, fx, FX, iyy, fy, FY);
            }
            __syncthreads();
            const int qs = t / FNPC, qr = t % FNPC;
            const bool one = t < spc * FNPC && r0 + qr < sm.queued[qs];
            if (one) {
                const int32_t *q = pts + 3 * sm.queue[qs][r0 + qr];
                double a1 = 0.0, a2 = 0.0, b1 = 0.0, b2 = 0.0;
                for (int k = 0; k < O.nlev; k++) {
                    a1 += O.amp_d[k] * sm.sh_d[0][k * spc + qs][qr] * O.vf_d[k];
                    a2 += O.amp_d[k] * sm.sh_d[0][(O.nlev + k) * spc + qs][qr] * O.vf_d[k];
                    b1 += O.amp_d[k] * sm.sh_d[1][k * spc + qs][qr] * O.vf_d[k];
                    b2 += O.amp_d[k] * sm.sh_d[1][(O.nlev + k) * spc + qs][qr] * O.vf_d[k];
                }
                const double x = (double)q[0] + ((a1 + a2) * O.vfac) * 4.0, z = (double)q[2] + ((b1 + b2) * O.vfac) * 4.0;
                sm.coord_d[qs][qr][0] = x;
                sm.coord_d[qs][qr][1] = z;
                sm.coord_d[qs][qr][2] = x * MG_SECOND_STACK;
                sm.coord_d[qs][qr][3] = z * MG_SECOND_STACK;
            }
            __syncthreads();
            if (active && own.noise != 0) {
                OffHdr x;
                x.ox = own.ox; x.oy = own.oy; x.oz = own.oz;
                lattice_header(x, true);
                const int n = min(sm.queued[ls] - r0, FNPC);
                for (int r = 0; r < n; r++) sm.val_d[t][r] = search_octave<false, double>(W, own, x, mine, sm.coord_d[ls][r]);
            }
            __syncthreads();
            if (one) {
                const int p = sm.queue[qs][r0 + qr];
                double v[MG_OW_NOISES - 1];
                for (int q = 1; q < MG_OW_NOISES; q++) {
                    const MgNoise &N = W.noise[q];
                    double a1 = 0.0, a2 = 0.0;
                    for (int k = 0; k < N.nlev; k++) a1 += N.amp_d[k] * sm.val_d[(N.base + k) * spc + qs][qr] * N.vf_d[k];
                    for (int k = 0; k < N.nlev; k++) a2 += N.amp_d[k] * sm.val_d[(N.base + N.nlev + k) * spc + qs][qr] * N.vf_d[k];
                    v[q - 1] = (a1 + a2) * N.vfac;
                }
                climate_finish_d(W, *spline, v[0], v[1], v[2], v[3], v[4], pts[3 * p + 1] * 4, targets + ((size_t)(s0 + qs) * np + p) * 6);
            }
        }
        __syncthreads(); /* every thread has read the lengths (the loop's last round) */
        if (t < FMAXS) sm.queued[t] = 0;
        __syncthreads();
    };

    auto within = [](const int32_t *q, int lim) { return q[0] > -lim && q[0] < lim && q[2] > -lim && q[2] < lim; };
    for (int p0 = 0; p0 < np; p0 += FNPC) {
        const int npc = min(FNPC, np - p0);
        __syncthreads(); /* lattices and headers complete / previous chunk consumed */
        /* ---- B: ShiftA (x, 0, z) and ShiftB (z, x, 0) octaves, item = (owner, point) */
        for (int item = t; item < nown * npc; item += FNT) {
            const int o = item % nown, p = item / nown, oj = o / spc;
            if (s0 + o % spc >= ns) continue;
            const auto &oh = sm.hdr[o];
            const IlvPerm<FPS> perm{pbase, o};
            const int32_t *pp = pts + 3 * (p0 + p);
            if (!within(pp, OT_COORD_LIM)) continue;
            const double f = O.freq[oj >= O.nlev ? oj - O.nlev : oj];
            double X = (double)pp[0], Z = (double)pp[2];
            if (oj >= O.nlev) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
            int ia, ib;
            int32_t ta, ua, tb, ub;
            ot_split_d(X, f, oh.ox, ia, ta, ua);
            ot_split_d(Z, f, oh.oz, ib, tb, ub);
            sm.sh[0][o][p] = ot_sample_d(perm, oh.iy, false, oh.fy, ia, ib, ta, ua, tb, ub);
            ot_split_d(Z, f, oh.ox, ia, ta, ua);
            ot_split_d(X, f, oh.oy, ib, tb, ub);
            sm.sh[1][o][p] = ot_sample_d(perm, oh.iz, true, oh.fz, ia, ib, ta, ua, tb, ub);
        }
        __syncthreads();
        /* ---- C: shifted coordinates of every (seed, point) */
        const int cs = t / FNPC, cp = t % FNPC;
        const bool item = t < spc * FNPC && cp < npc && s0 + cs < ns;
        const int32_t *pp = pts + 3 * (p0 + (item ? cp : 0));
        const bool skip = !within(pp, OT_COORD_LIM);
        if (item) {
            int64_t sa = 0, sb = 0; /* units of 2^-59 */
            for (int k = 0; k < O.nlev; k++) {
                const int64_t va = sm.sh[0][k * spc + cs][cp] + sm.sh[0][(O.nlev + k) * spc + cs][cp];
                const int64_t vb = sm.sh[1][k * spc + cs][cp] + sm.sh[1][(O.nlev + k) * spc + cs][cp];
                sa = ot_madw((int32_t)(va >> 31), O.c30[k], sa);
                sb = ot_madw((int32_t)(vb >> 31), O.c30[k], sb);
            }
            const int64_t x = skip ? 0 : ((int64_t)pp[0] << 32) + (sa >> 25), z = skip ? 0 : ((int64_t)pp[2] << 32) + (sb >> 25);
            sm.coord[cs][cp][0] = x;
            sm.coord[cs][cp][1] = z;
            sm.coord[cs][cp][2] = x + __mul64hi(x, OT_STACK_C);
            sm.coord[cs][cp][3] = z + __mul64hi(z, OT_STACK_C);
        }
        const bool any = __syncthreads_or(item && !skip); /* else every point of the chunk is for the queues */
        /* ---- D: climate octaves, each thread on its own lattice */
        if (any && active && own.noise != 0) {
            for (int p = 0; p < npc; p++) {
                const int64_t sx = (sm.coord[ls][p][own.st ? 2 : 0] >> lev) + oxq, sz = (sm.coord[ls][p][own.st ? 3 : 1] >> lev) + ozq;
                sm.val[t][p] = ot_sample_d(mine, iy, false, fix, ot_hi(sx), ot_hi(sz), (int32_t)((uint32_t)sx >> 1), ot_fade31((uint32_t)sx),
                                           (int32_t)((uint32_t)sz >> 1), ot_fade31((uint32_t)sz));
            }
        }
        __syncthreads();
        /* ---- E: the five noises */
        if (item) {
#pragma unroll
            for (int q = 1; q < MG_OW_NOISES; q++) {
                const MgNoise &N = W.noise[q];
                int64_t acc = 0;
                for (int k = 0; k < N.nlev; k++) {
                    const int64_t l = sm.val[(N.base + k) * spc + cs][cp] + sm.val[(N.base + N.nlev + k) * spc + cs][cp];
                    acc = ot_madw((int32_t)(l >> 31), N.c30[k], acc);
                }
                sm.v[cs][(p0 + cp) % TQ_CAP][q - 1] = (int32_t)(acc >> 30);
            }
        }
        const int done = p0 + npc, from = (done - 1) / TQ_CAP * TQ_CAP; /* points [from, done) have values */
        if (done != np && done % TQ_CAP) continue;
        __syncthreads();
        /* ---- F: the targets that they may have */
        for (int i = t; i < spc * (done - from); i += FNT) {
            const int s = i / (done - from), p = from + i % (done - from);
            if (s0 + s >= ns) continue;
            const int32_t *q = pts + 3 * p;
            const bool out17 = !within(q, (1 << 17) - OT_W);
            int32_t v[MG_OW_NOISES - 1], ta[6], tb[6], eq[MG_OW_NOISES];
#pragma unroll
            for (int k = 1; k < MG_OW_NOISES; k++) {
                v[k - 1] = sm.v[s][p - from][k - 1];
                eq[k] = out17 ? W.noise[k].tile_eq_far : W.noise[k].tile_eq;
            }
            float es;
            ot_climate_targets(W, *spline, v, eq, (int32_t)__double2ll_rn((depth_grad_d(W, q[1] * 4) + W.off_d) * 0x1.0p28), ta, tb, es);
            bool ok = es < 1.0f && within(q, OT_COORD_LIM);
#pragma unroll
            for (int k = 0; k < 6; k++) ok &= ta[k] == tb[k];
            if (ok) {
                int32_t *o = targets + ((size_t)(s0 + s) * np + p) * 6;
#pragma unroll
                for (int k = 0; k < 6; k++) o[k] = ta[k];
            } else {
                sm.queue[s][atomicAdd(&sm.queued[s], 1)] = p;
            }
        }
        drain();
    }
}
/* samples of a warp in the tree kernels, whose lanes' targets it takes one after another: fewer than 32 when there are too few
 * samples to fill the chip with warps of 32 (49,533 samples: 106 -> 88 us) */
static int tree_lanes(long long n) {
    const long long k = (n + 152 * 40 - 1) / (152 * 40);
    return k < 32 ? (int)k : 32;
}
/* the tree for samples whose targets are known */
__global__ void __launch_bounds__(128) k_ow_targets_tree(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                         const int32_t *__restrict__ tg, long long n, int lanes,
                                                         uint8_t *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const long long g = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * lanes + lane;
    const bool in = lane < lanes && g < n;
    int32_t t[6] = {0, 0, 0, 0, 0, 0};
    if (in)
        for (int k = 0; k < 6; k++) t[k] = tg[g * 6 + k];
    const int leaf = tree_search_lanes(tree, W, t, in);
    if (in) out[g] = tree[leaf].biome;
}
/* Finish the climate of every sample from its five noise values (ridges_folded, offset spline, depth,
 * quantisation; engine/mc_climate.h:126-170) and search the R-tree (ENGINE rule). One thread per sample. */
template <bool FM>
__global__ void __launch_bounds__(128) k_ow_finish_tree(const __grid_constant__ MgWorldDesc W,
                                                        const MgTreeNode *__restrict__ tree,
                                                        const typename std::conditional<FM, float, double>::type *__restrict__ clim,
                                                        int ns, const int32_t *__restrict__ pts, int np, int lanes,
                                                        uint8_t *__restrict__ out, int32_t *__restrict__ targets) {
    __shared__ MgSpline S;
    {
        const uint4 *c = reinterpret_cast<const uint4 *>(&W.spline);
        uint4 *d = reinterpret_cast<uint4 *>(&S);
        for (int i = threadIdx.x; i < (int)(sizeof(MgSpline) / 16); i += blockDim.x) d[i] = c[i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long g = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * lanes + lane;
    const bool in = lane < lanes && g < (long long)ns * np;
    int32_t tg[6] = {0, 0, 0, 0, 0, 0};
    if (in) {
        const int p = (int)(g % np);
        const int by = pts[3 * p + 1] * 4;
        const auto *v = clim + (size_t)g * 5;
        if (FM) climate_finish_f(W, S, (float)v[0], (float)v[1], (float)v[2], (float)v[3], (float)v[4], by, tg);
        else climate_finish_d(W, S, (double)v[0], (double)v[1], (double)v[2], (double)v[3], (double)v[4], by, tg);
    }
    const int leaf = tree_search_lanes(tree, W, tg, in);
    if (!in) return;
    out[g] = tree[leaf].biome;
    if (targets)
        for (int k = 0; k < 6; k++) targets[g * 6 + k] = tg[k];
}

/* ---- seed search, Overworld, one observation of every candidate (engine/cuda/mc_gpu.cuh:476-493, stage [0]), in three kernels.
 * The shuffles bound it (46 of 256 steps per candidate, the integer pipe), so it builds no more lattices than decide a candidate:
 * k_ow_search_th those of the offset, temperature and humidity (14 of 46), after which a table (k_search_possible) says whether
 * any leaf with an observed biome can still be nearest (about 29 % of the candidates); k_ow_search_rest the others' for those,
 * k_ow_search_first the target and the tree.  2^20 candidates: 14.7 + 0.9 ms in one stage, 8.6 ms in three. */

/* possible[r] bit c: a leaf with a biome of the mask can be nearest to a target of temperature class r and humidity class c
 * (class: cuts at or below the value).  It cannot when some other leaf holds the whole class while it does not, and holds its box
 * in every other dimension: then that leaf is closer, whatever the other coordinates.  One block per leaf (a warp per leaf took 75 us,
 * a chain of loads). */
__global__ void __launch_bounds__(256) k_search_possible(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                         MgObs o, uint32_t *__restrict__ possible) {
    const int lane = threadIdx.x & 31;
    const MgTreeNode *L = tree + W.leaf_off;
    auto cls = [&](int d, int v) {
        int k = 0;
        for (int i = 0; i < W.cuts[d]; i++) k += W.cut[d][i] <= v;
        return k;
    };
    auto bits = [](int a, int b) { return b < a ? 0u : (0xFFFFFFFFu >> (31 - (b - a))) << a; };
    if (W.cuts[0] < 0 || W.cuts[1] < 0) { /* too many bounds for the table: everything is possible */
        if (blockIdx.x == 0 && threadIdx.x < 32) possible[threadIdx.x] = 0xFFFFFFFFu;
        return;
    }
    __shared__ uint32_t row[32];
    {
        const MgTreeNode n = L[blockIdx.x];
        if (!obs_in(o, n.biome)) return;
        if (threadIdx.x < 32) row[threadIdx.x] = 0;
        __syncthreads();
        uint32_t covered = 0; /* of row `lane` */
        for (int m0 = (int)(threadIdx.x & ~31u); m0 < W.tree_leaves; m0 += (int)blockDim.x) {
            bool over = m0 + lane < W.tree_leaves;
            const MgTreeNode m = L[over ? m0 + lane : 0];
            for (int d = 2; d < 6; d++) over &= m.lo[d] <= n.lo[d] && m.nhi[d] <= n.nhi[d];
            over &= m.d7 <= n.d7;
            for (unsigned w = __ballot_sync(0xFFFFFFFFu, over); w; w &= w - 1) {
                const MgTreeNode &c = L[m0 + __ffs((int)w) - 1];
                if (lane >= cls(0, c.lo[0]) && lane <= cls(0, -c.nhi[0])) covered |= bits(cls(1, c.lo[1]), cls(1, -c.nhi[1]));
            }
        }
        atomicOr(&row[lane], covered);
        __syncthreads();
        if (threadIdx.x >= 32) return;
        const uint32_t own = lane >= cls(0, n.lo[0]) && lane <= cls(0, -n.nhi[0]) ? bits(cls(1, n.lo[1]), cls(1, -n.nhi[1])) : 0u;
        atomicOr(&possible[lane], own | ~row[lane]);
    }
}

/* candidates that are left after the first stage: their index, shifted coordinates and (in clim) first two noise values */
template <typename V>
struct SearchList {
    unsigned *count;
    int32_t *index;
    double2 *coord;
    V *clim; /* 5 per entry */
};
template <typename V>
struct SearchSmem {
    uint32_t perm[64][FPS];
    V val[FPS], valb[FPS]; /* octave values by owner */
    double coord[FPS / 2][4];
};
template <bool FM>
__global__ void __launch_bounds__(FPS) k_ow_search_th(const __grid_constant__ MgWorldDesc W, const int64_t *__restrict__ seeds, int ns,
                                                      const int32_t *__restrict__ pts, const uint32_t *__restrict__ possible,
                                                      SearchList<typename std::conditional<FM, float, double>::type> out,
                                                      unsigned long long *__restrict__ fail) {
    typedef typename std::conditional<FM, float, double>::type V;
    extern __shared__ uint4 smem_raw[];
    SearchSmem<V> &sm = *reinterpret_cast<SearchSmem<V> *>(smem_raw);
    const int t = threadIdx.x, nt = W.noise[3].base, spc = FPS / nt, s0 = blockIdx.x * spc, ls = t % spc;
    const bool active = t / spc < nt && s0 + ls < ns;
    FusedOwn own;
    OffHdr h;
    if (active) {
        fused_lattice(W, seeds[s0 + ls], t / spc, &sm.perm[0][t], own);
        h.ox = own.ox; h.oy = own.oy; h.oz = own.oz;
        lattice_header(h, !FM);
    }
    const IlvPerm<FPS> perm{reinterpret_cast<const uint8_t *>(&sm.perm[0][0]), t};
    const MgNoise &O = W.noise[0];
    if (active && own.noise == 0) { /* ShiftA (x, 0, z) and ShiftB (z, x, 0) */
        const int32_t *pp = pts + (size_t)(s0 + ls) * 3;
        double X = (double)pp[0], Z = (double)pp[2];
        if (own.st) { X = X * MG_SECOND_STACK; Z = Z * MG_SECOND_STACK; }
        const double f = O.freq[own.lev];
        const int k = O.fexp[own.lev];
        int ix, iz, iy;
        if constexpr (FM) {
            float fx, fz, fy;
            split_fk(X, f, k, own.ox, ix, fx);
            split_fk(Z, f, k, own.oz, iz, fz);
            sm.val[t] = (V)octave_y0<float>(perm, h, ix, fx, iz, fz);
            split_fk(Z, f, k, own.ox, ix, fx);
            split_fk(X, f, k, own.oy, iy, fy);
            sm.valb[t] = (V)octave_z0<float>(perm, h, ix, fx, iy, fy);
        } else {
            double fx, fz, fy;
            int64_t FX, FZ, FY;
            split_dk(X, f, k, own.ox, ix, fx, FX);
            split_dk(Z, f, k, own.oz, iz, fz, FZ);
            sm.val[t] = (V)octave_d_y0(perm, h, ix, fx, FX, iz, fz, FZ);
            split_dk(Z, f, k, own.ox, ix, fx, FX);
            split_dk(X, f, k, own.oy, iy, fy, FY);
            sm.valb[t] = (V)octave_d_z0(perm, h, ix, fx, FX, iy, fy, FY);
        }
    }
    __syncthreads();
    const bool mine = t < spc && s0 + t < ns;
    double2 at = make_double2(0.0, 0.0);
    if (mine) {
        const int32_t *pp = pts + (size_t)(s0 + t) * 3;
        at.x = (double)pp[0] + (double)(search_sum<FM, V>(O, sm.val, 0, spc, t) * (V)4.0);
        at.y = (double)pp[2] + (double)(search_sum<FM, V>(O, sm.valb, 0, spc, t) * (V)4.0);
        sm.coord[t][0] = at.x;
        sm.coord[t][1] = at.y;
        sm.coord[t][2] = at.x * MG_SECOND_STACK;
        sm.coord[t][3] = at.y * MG_SECOND_STACK;
    }
    __syncthreads();
    if (active && own.noise != 0) sm.val[t] = search_octave<FM, V>(W, own, h, perm, sm.coord[ls]);
    __syncthreads();
    if (t < 32 * ((spc + 31) / 32)) {
        bool left = false;
        V th[2] = {0, 0};
        if (mine) {
            int c[2] = {0, 0};
            for (int d = 0; d < 2; d++) {
                th[d] = search_sum<FM, V>(W.noise[1 + d], sm.val, W.noise[1 + d].base, spc, t);
                const int v = quantize((float)th[d]);
                for (int i = 0; i < W.cuts[d]; i++) c[d] += W.cut[d][i] <= v;
            }
            left = possible[c[0]] >> c[1] & 1;
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, left), f = __ballot_sync(0xFFFFFFFFu, mine && !left);
        unsigned k = 0;
        if ((t & 31) == 0) {
            if (m) k = atomicAdd(out.count, (unsigned)__popc(m));
            if (f) atomicAdd(fail, (unsigned long long)__popc(f));
        }
        k = __shfl_sync(0xFFFFFFFFu, k, 0) + (unsigned)__popc(m & ((1u << (t & 31)) - 1));
        if (left) {
            out.index[k] = s0 + t;
            out.coord[k] = at;
            out.clim[(size_t)k * 5] = th[0];
            out.clim[(size_t)k * 5 + 1] = th[1];
        }
    }
}
/* the other three noises of the candidates in the list */
template <bool FM>
__global__ void __launch_bounds__(FPS) k_ow_search_rest(const __grid_constant__ MgWorldDesc W, const int64_t *__restrict__ seeds,
                                                        SearchList<typename std::conditional<FM, float, double>::type> list) {
    typedef typename std::conditional<FM, float, double>::type V;
    extern __shared__ uint4 smem_raw[];
    SearchSmem<V> &sm = *reinterpret_cast<SearchSmem<V> *>(smem_raw);
    const int t = threadIdx.x, j0 = W.noise[3].base, nt = W.ntables - j0, spc = FPS / nt, ls = t % spc;
    const int ns = (int)*list.count;
    const IlvPerm<FPS> perm{reinterpret_cast<const uint8_t *>(&sm.perm[0][0]), t};
    for (int s0 = (int)blockIdx.x * spc; s0 < ns; s0 += (int)gridDim.x * spc) {
        if (t < spc && s0 + t < ns) {
            const double2 at = list.coord[s0 + t];
            sm.coord[t][0] = at.x;
            sm.coord[t][1] = at.y;
            sm.coord[t][2] = at.x * MG_SECOND_STACK;
            sm.coord[t][3] = at.y * MG_SECOND_STACK;
        }
        __syncthreads();
        if (t / spc < nt && s0 + ls < ns) {
            FusedOwn own;
            OffHdr h;
            fused_lattice(W, seeds[list.index[s0 + ls]], j0 + t / spc, &sm.perm[0][t], own);
            h.ox = own.ox; h.oy = own.oy; h.oz = own.oz;
            lattice_header(h, !FM);
            sm.val[t] = search_octave<FM, V>(W, own, h, perm, sm.coord[ls]);
        }
        __syncthreads();
        if (t < 3 * spc) {
            const int q = 3 + t / spc, s = t % spc;
            if (s0 + s < ns) list.clim[(size_t)(s0 + s) * 5 + q - 1] = search_sum<FM, V>(W.noise[q], sm.val, W.noise[q].base - j0, spc, s);
        }
        __syncthreads();
    }
}
/* the target and the tree; passing candidates are appended to `surv`, failures counted into *fail */
template <bool FM>
__global__ void __launch_bounds__(128) k_ow_search_first(const __grid_constant__ MgWorldDesc W, const MgTreeNode *__restrict__ tree,
                                                         SearchList<typename std::conditional<FM, float, double>::type> list,
                                                         const int64_t *__restrict__ seeds, const int32_t *__restrict__ pts, MgObs o,
                                                         int ties, int64_t *__restrict__ surv, unsigned *__restrict__ nsurv,
                                                         unsigned long long *__restrict__ fail) {
    __shared__ MgSpline S;
    {
        const uint4 *c = reinterpret_cast<const uint4 *>(&W.spline);
        uint4 *d = reinterpret_cast<uint4 *>(&S);
        for (int i = threadIdx.x; i < (int)(sizeof(MgSpline) / 16); i += blockDim.x) d[i] = c[i];
    }
    __syncthreads();
    const int n = (int)*list.count, lane = threadIdx.x & 31, warps = (int)(gridDim.x * blockDim.x) >> 5;
    const int lanes = min((n + warps - 1) / warps, 32); /* (tree_lanes) */
    int nf = 0;
    for (int b = (int)blockIdx.x * 4 * lanes; b < n; b += warps * lanes) {
        const int k = b + (int)(threadIdx.x >> 5) * lanes + lane;
        const bool in = lane < lanes && k < n;
        const int g = in ? list.index[k] : 0;
        int32_t tg[6] = {0, 0, 0, 0, 0, 0};
        if (in) {
            const auto *v = list.clim + (size_t)k * 5;
            const int by = pts[3 * (size_t)g + 1] * 4;
            if (FM) climate_finish_f(W, S, (float)v[0], (float)v[1], (float)v[2], (float)v[3], (float)v[4], by, tg);
            else climate_finish_d(W, S, (double)v[0], (double)v[1], (double)v[2], (double)v[3], (double)v[4], by, tg);
        }
        const bool met = obs_accept(o, tree, W, tg, ties != 0, in);
        if (met) surv[atomicAdd(nsurv, 1u)] = seeds[g];
        nf += __syncthreads_count(in && !met);
    }
    if (threadIdx.x == 0 && nf) atomicAdd(fail, (unsigned long long)nf);
}

/* scratch: the table, the list's counter, index, coordinates and noise values */
size_t search_scratch_bytes(const MgWorldDesc &W, long long n) {
    return 256 + (size_t)n * (sizeof(double2) + 5 * (W.fmode ? sizeof(float) : sizeof(double)) + sizeof(int32_t));
}
template <bool FM>
static int search_first_t(const MgWorldDesc &W, const MgTreeNode *tree, const int64_t *seeds, int ns, const int32_t *pts,
                          const MgObs &o, int ties, void *scratch, int64_t *surv, unsigned *nsurv,
                          unsigned long long *fail, cudaStream_t st) {
    typedef typename std::conditional<FM, float, double>::type V;
    const int sm = (int)sizeof(SearchSmem<V>);
    cudaError_t e = cudaFuncSetAttribute(k_ow_search_th<FM>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (!e) e = cudaFuncSetAttribute(k_ow_search_rest<FM>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (!e) e = cudaFuncSetAttribute(k_ow_search_th<FM>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (!e) e = cudaFuncSetAttribute(k_ow_search_rest<FM>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    uint8_t *p = (uint8_t *)scratch;
    uint32_t *possible = (uint32_t *)p;
    SearchList<V> list;
    list.count = (unsigned *)(p + 128);
    list.coord = (double2 *)(p + 256);
    list.clim = (V *)(list.coord + ns);
    list.index = (int32_t *)(list.clim + (size_t)ns * 5);
    if (!e) e = cudaMemsetAsync(p, 0, 256, st);
    if (e) return (int)e;
    {
        ProfScope ps_(K_SEARCH_CELLS, st);
        k_search_possible<<<(unsigned)W.tree_leaves, 256, 0, st>>>(W, tree, o, possible);
    }
    count_launch_external();
    const int spc = FPS / W.noise[3].base;
    {
        ProfScope ps_(K_OW_SEED_CLIMATE, st);
        k_ow_search_th<FM><<<(unsigned)((ns + spc - 1) / spc), FPS, sm, st>>>(W, seeds, ns, pts, possible, list, fail);
    }
    count_launch_external();
    {
        ProfScope ps_(K_OW_SEED_CLIMATE, st);
        k_ow_search_rest<FM><<<4 * 152, FPS, sm, st>>>(W, seeds, list);
    }
    count_launch_external();
    {
        ProfScope ps_(K_SEARCH_FIRST, st);
        k_ow_search_first<FM><<<8 * 152, 128, 0, st>>>(W, tree, list, seeds, pts, o, ties, surv, nsurv, fail);
    }
    count_launch_external();
    return 0;
}

int launch_ow_search_first(const MgWorldDesc &W, const MgTreeNode *tree, const int64_t *seeds, int ns, const int32_t *pts,
                           const MgObs &o, int ties, void *scratch, int64_t *surv, unsigned *nsurv,
                           unsigned long long *fail, cudaStream_t st) {
    if (ns <= 0) return 0;
    int rc = W.fmode ? search_first_t<true>(W, tree, seeds, ns, pts, o, ties, scratch, surv, nsurv, fail, st)
                     : search_first_t<false>(W, tree, seeds, ns, pts, o, ties, scratch, surv, nsurv, fail, st);
    return rc ? rc : (int)cudaGetLastError();
}

bool fused_supported(const MgWorldDesc &W) {
    if (W.dim != MG_OVERWORLD || W.ntables > FMAXT || W.noise[0].base != 0) return false;
    const int spc = FNT / W.ntables;
    return spc >= 1 && spc <= FMAXS && 2 * W.noise[0].nlev * spc <= FMAXOFF;
}
size_t fused_scratch_bytes(const MgWorldDesc &W, long long samples) {
    return (size_t)samples * 5 * (W.fmode ? sizeof(float) : sizeof(double));
}

template <bool FM>
static int fused_t(const MgWorldDesc &W, const MgTreeNode *tree, const int64_t *seeds, int ns, const int32_t *pts, int np,
                   uint8_t *out, int32_t *tg, void *scratch, cudaStream_t st) {
    typedef typename std::conditional<FM, float, double>::type V;
    const size_t sm = sizeof(FusedSmem<V>);
    cudaError_t e = cudaFuncSetAttribute(k_ow_seed_climate<FM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (!e) e = cudaFuncSetAttribute(k_ow_seed_climate<FM>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared); /* room for 4 CTAs per SM */
    if (e) return (int)e;
    const int spc = FNT / W.ntables;
    V *clim = (V *)scratch;
    {
        ProfScope ps_(K_OW_SEED_CLIMATE, st);
        k_ow_seed_climate<FM><<<(unsigned)((ns + spc - 1) / spc), FNT, sm, st>>>(W, seeds, ns, pts, np, clim);
    }
    count_launch_external();
    const long long n = (long long)ns * np;
    {
        ProfScope ps_(K_OW_FINISH_TREE, st);
        const int lanes = tree_lanes(n);
        k_ow_finish_tree<FM><<<(unsigned)((n + 4 * lanes - 1) / (4 * lanes)), 128, 0, st>>>(W, tree, clim, ns, pts, np, lanes, out, tg);
    }
    count_launch_external();
    return 0;
}

/* the double branch in fixed point: targets into tg, or the scratch */
static int targets_t(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const int64_t *seeds, int ns, const int32_t *pts,
                     int np, uint8_t *out, int32_t *tg, cudaStream_t st) {
    const int sm = (int)sizeof(TargetSmem);
    cudaError_t e = cudaFuncSetAttribute(k_ow_seed_targets, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (!e) e = cudaFuncSetAttribute(k_ow_seed_targets, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e) return (int)e;
    const int spc = FNT / W.ntables;
    {
        ProfScope ps_(K_OW_SEED_CLIMATE, st);
        k_ow_seed_targets<<<(unsigned)((ns + spc - 1) / spc), FNT, sm, st>>>(W, &d_world->spline, seeds, ns, pts, np, tg);
    }
    count_launch_external();
    const long long n = (long long)ns * np;
    {
        ProfScope ps_(K_OW_FINISH_TREE, st);
        const int lanes = tree_lanes(n);
        k_ow_targets_tree<<<(unsigned)((n + 4 * lanes - 1) / (4 * lanes)), 128, 0, st>>>(W, tree, tg, n, lanes, out);
    }
    count_launch_external();
    return 0;
}

int launch_ow_seed_points(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const int64_t *seeds, int ns,
                          const int32_t *pts, int np, uint8_t *out, int32_t *tg, void *scratch, cudaStream_t st) {
    if ((long long)ns * np <= 0) return 0;
    if (!W.fmode && ow_tile_supported(W)) {
        const int r = targets_t(W, d_world, tree, seeds, ns, pts, np, out, tg ? tg : (int32_t *)scratch, st);
        return r ? r : (int)cudaGetLastError();
    }
    int rc = W.fmode ? fused_t<true>(W, tree, seeds, ns, pts, np, out, tg, scratch, st)
                     : fused_t<false>(W, tree, seeds, ns, pts, np, out, tg, scratch, st);
    return rc ? rc : (int)cudaGetLastError();
}

}  // namespace mg
