/* launch.h -- host launchers of the biome kernels (kernels.cu), called by the C ABI (api.cpp).
 * All return a cudaError_t value (0 on success) and enqueue on `st` without synchronising. */
#ifndef MG_LAUNCH_H
#define MG_LAUNCH_H
#include <cuda_runtime.h>
#include <stddef.h>

#include "mg_types.h"

namespace mg {

/* GRID_CHAIN and CHUNK_ORDER: a cell's target, its first minimum leaf (a node index), fitness and tie flag */
struct ChainRec { int32_t tg[6]; uint64_t d; int32_t leaf; int32_t tie; };

long long launch_count();
void count_launch_external(); /* for launchers outside kernels.cu */

/* per-seed lattices: d_states[s * W.ntables + j] */
int launch_setup(const MgWorldDesc &W, const int64_t *d_seeds, int ns, MgLattice *d_states, cudaStream_t st);

/* seeds x quart points, ENGINE rule (targets optional) */
int launch_points(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *states, int ns, const int32_t *pts,
                  int np, uint8_t *out, int32_t *targets, cudaStream_t st);

/* seeds x points for the Overworld (fused.cu): lattices built and sampled in shared memory by one kernel,
 * climate finish + R-tree by a second.  Scratch: fused_scratch_bytes(W, ns * np) (five noise values per
 * sample).  fused_supported() tells whether a world's lattice count fits the kernel. */
bool fused_supported(const MgWorldDesc &W);
size_t fused_scratch_bytes(const MgWorldDesc &W, long long samples);
int launch_ow_seed_points(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const int64_t *seeds, int ns,
                          const int32_t *pts, int np, uint8_t *out, int32_t *targets, void *scratch, cudaStream_t st);

/* seed search, Overworld, one observation (one quart cell per candidate at pts[3i..3i+2]): candidates
 * that pass go to surv (count *nsurv), failures are added to *fail.  Scratch: search_scratch_bytes(W, ns). */
size_t search_scratch_bytes(const MgWorldDesc &W, long long n);
int launch_ow_search_first(const MgWorldDesc &W, const MgTreeNode *tree, const int64_t *seeds, int ns, const int32_t *pts,
                           const MgObs &o, int ties, void *scratch, int64_t *surv, unsigned *nsurv,
                           unsigned long long *fail, cudaStream_t st);

/* one seed's quart grid.  d_world: the description's device copy.  Scratch: quart_scratch_bytes. */
size_t quart_scratch_bytes(const MgWorldDesc &W, int rule, int nx, int nz);
bool quart_scratch_optional(const MgWorldDesc &W, int rule); /* may be null when there is no memory for it */
int launch_quart_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int qx0, int qz0,
                      int nx, int nz, int qy, int rule, uint8_t *out, void *scratch, cudaStream_t st);

/* block-coordinate biomes (zoom + chunk-cell ties): a grid when xyz == nullptr, else nx points at xyz
 * (nz == 1).  d_world: the description's device copy.  Scratch: block_scratch_bytes; for the End the chunk classes of
 * [ecx0, ecx0+encx) x [ecz0, ecz0+encz), or null to evaluate the class per sample. */
size_t block_scratch_bytes(const MgWorldDesc &W, int x0, int z0, int nx, int nz, bool points);
int launch_block_biomes(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int64_t zseed,
                        int x0, int z0, int nx, int nz, int step, int y, const int32_t *xyz, uint8_t *out, void *scratch,
                        int ecx0, int ecz0, int encx, int encz, cudaStream_t st);

/* a few block points (host coordinates) of the worlds that block_few_supported takes */
#define FEW_POINTS 64
bool block_few_supported(const MgWorldDesc &W, int n);
int launch_block_few(const MgWorldDesc &W, const MgTreeNode *tree, const MgLattice *state, int64_t zseed, const int32_t *xyz, int n,
                     uint8_t *out, cudaStream_t st);

/* the same through the tile kernels (owtile.cu), for worlds ow_tile_supported takes.  rec: the
 * cells' chain records, or null.  Scratch: ow_grid_scratch_bytes. */
bool ow_block_grid_supported(const MgWorldDesc &W, int x0, int z0);
size_t ow_grid_scratch_bytes(const MgWorldDesc &W, bool chunk_rule, long long cells);
int launch_ow_quart_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int qx0,
                         int qz0, int nx, int nz, int qy, ChainRec *rec, uint8_t *out, void *scratch, cudaStream_t st);
int launch_ow_block_grid(const MgWorldDesc &W, const MgWorldDesc *d_world, const MgTreeNode *tree, const MgLattice *state, int64_t zseed,
                         int x0, int z0, int nx, int nz, int step, int y, const int32_t *xyz, uint8_t *out, void *scratch,
                         cudaStream_t st);

/* Overworld density functions (continents, erosion, ridges, offset, depth) at n block points xyz[3i..3i+2] of
 * one seed's lattices: out[5i + k] (cudaErrorInvalidValue for other dimensions) */
int launch_density(const MgWorldDesc &W, const MgLattice *state, int n, const int32_t *xyz, double *out, cudaStream_t st);

/* pipe microbenchmarks (pipes.cu) */
int pipe_rate(int pipe, double *gops);

}  // namespace mg
#endif
