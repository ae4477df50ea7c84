/* legacy.cuh -- lattices built from java.util.Random: the Nether's noises and the End's simplex, one permutation column per thread
 * (byte i at column + (i >> 2) * 4 ROW + (i & 3)). */
#ifndef MG_LEGACY_CUH
#define MG_LEGACY_CUH
#include "device.cuh"

namespace mg {
using namespace mgd;

/* one lattice's offsets and permutation from the state, which then is the next lattice's; returns the rejected draws */
template <int ROW>
__device__ __noinline__ int legacy_octave(uint64_t &s, uint32_t *col, MgLattice &h) {
    h.ox = lcg_double(s) * 256.0;
    h.oy = lcg_double(s) * 256.0;
    h.oz = lcg_double(s) * 256.0;
    for (int w = 0; w < 64; w++) col[w * ROW] = 0x03020100u + 0x04040404u * (uint32_t)w;
    return lcg_shuffle<ROW>(reinterpret_cast<uint8_t *>(col), s);
}

/* A Nether noise of a seed: each stack builds the zero octave first, then octaves zero-1 .. 0, skipping 262 draws for an absent one
 * (engine/mc_noise.h:266-282, engine/cuda/mcg_host.c:49-51); noise n's generator is seeded with seed + n.  A built octave takes 262
 * draws too and those it rejects (4e-6 an octave), so a noise's octaves are built at once by LEGACY_GROUP neighbouring lanes, each
 * from the state that many draws on; those after a rejection once more, from the state moved on by it.  Six shuffles in a row, 31 us
 * each, were the latency of a small batch: 187 -> 45 us.  A noise with more octaves than lanes is built by the first lane.
 * store(i, h) writes lattice i of the noise from the calling thread's column.  All lanes of the group call it. */
#define LEGACY_GROUP 6 /* the game's: three octaves in each of two stacks */
#define LEGACY_PER_WARP (32 / LEGACY_GROUP)
/* threads for n noises, in whole blocks' warps; the noise of this thread (its group's), or -1 */
__host__ __device__ inline long long legacy_threads(long long n) { return (n + LEGACY_PER_WARP - 1) / LEGACY_PER_WARP * 32; }
__device__ __forceinline__ long long legacy_index(long long thread) {
    const int lane = (int)(thread & 31);
    return lane < LEGACY_GROUP * LEGACY_PER_WARP ? (thread >> 5) * LEGACY_PER_WARP + lane / LEGACY_GROUP : -1;
}
template <int ROW, typename STORE>
__device__ __forceinline__ void legacy_noise(const MgNoise &N, int n, int64_t seed, uint32_t *col, const STORE &store) {
    const int gl = (threadIdx.x & 31) % LEGACY_GROUP, first = (threadIdx.x & 31) - gl;
    const unsigned group = ((1u << LEGACY_GROUP) - 1) << first;
    const uint64_t st = lcg_init((int64_t)((uint64_t)seed + (uint64_t)n));
    const int zero = -N.first;
    auto level = [&](int q) { /* of octave q, or -1 */
        int k = N.nlev - 1;
        while (k >= 0 && N.idx[k] != q) k--;
        return q >= 0 && q < N.octs ? k : -1;
    };
    int unit = 0, at = 0, lattice = -1; /* the octaves built, counted; mine: draws before it, its lattice or -1 */
    for (int stack = 0; stack < 2; stack++)
        for (int q = zero; q >= 0 || q == zero; q--) {
            const int k = level(q);
            if (q != zero && k < 0) continue;
            if (unit == gl) {
                at = 262 * (stack * (max(zero, 0) + 1) + zero - q);
                lattice = k >= 0 ? stack * N.nlev + k : -1;
            }
            unit++;
        }
    MgLattice h;
    if (unit <= LEGACY_GROUP) {
        int moved = -1, rejected = 0, before = 0; /* draws that the octaves before this one rejected: taken, found */
        while (__ballot_sync(group, gl < unit && before != moved) & group) {
            if (gl < unit && before != moved) {
                uint64_t s = lcg_jump(st, (uint32_t)(at + before));
                rejected = legacy_octave<ROW>(s, col, h);
                moved = before;
            }
            before = 0;
            for (int k = 0; k < LEGACY_GROUP - 1; k++) {
                const int r = __shfl_sync(group, rejected, first + k);
                if (k < gl) before += r;
            }
        }
        if (gl < unit && lattice >= 0) store(lattice, h);
        return;
    }
    if (gl) return;
    uint64_t s = st;
    for (int stack = 0; stack < 2; stack++)
        for (int q = zero; q >= 0 || q == zero; q--) {
            const int k = level(q);
            if (q != zero && k < 0) {
                s = lcg_jump(s, 262);
                continue;
            }
            legacy_octave<ROW>(s, col, h);
            if (k >= 0) store(stack * N.nlev + k, h);
        }
}
/* End: LegacyRandomSource(seed).consumeCount(17292), then the simplex lattice (engine/mc_end.h:18-22) */
template <int ROW>
__device__ __forceinline__ void legacy_end(int64_t seed, uint32_t *col, MgLattice &h) {
    uint64_t s = lcg_jump(lcg_init(seed), 17292);
    legacy_octave<ROW>(s, col, h);
}

}  // namespace mg
#endif
