/* batch.h -- device layouts and launchers of the batched (many requests, one launch) form. */
#ifndef MG_BATCH_H
#define MG_BATCH_H
#include <cuda_runtime.h>
#include <stdint.h>

#include "mg_types.h"

/* one request of a batch: a quart-resolution region of one (world, seed) */
typedef struct {
    int32_t world;   /* index into the batch's world table */
    int32_t state;   /* first lattice of its seed in the state pool */
    int32_t qx0, qz0, nx, nz, qy;
    int32_t tie;     /* MG_TIE_ENGINE or MG_TIE_CHUNK_CELL */
    int64_t tile0;   /* number of the request's first tile */
    int64_t out_off; /* its first output byte */
} MgBatchReq;

/* one (world, seed) whose lattices the setup kernels write at pool[slot ...] */
typedef struct {
    int64_t seed;
    int32_t world;
    int32_t slot;
} MgSetupEntry;

#define BATCH_SHAPES 4
/* The requests of a batch come in three groups, each contiguous and with a tile numbering of its own: Overworld
 * requests that the tile kernels take by branch (owtile.cu: 16 x 16-cell tiles), then everything else (batch.cu). */
enum { BATCH_OW_D = 0, BATCH_OW_F = 1, BATCH_REST = 2, BATCH_GROUPS = 3 };
namespace mg {
struct BatchGroups {
    int n[BATCH_GROUPS];
    long long tiles[BATCH_GROUPS];
};
/* device counters of a batch: tiles taken per group, cells recorded as open per Overworld group */
#define BATCH_COUNTERS (BATCH_GROUPS + 2)
/* the group of a world's requests, and of one of them */
int batch_world_group(const MgWorldDesc &W, int tie);
int batch_group(int world_group, int qx0, int qz0, int nx, int nz);

/* ---- owtile.cu: worlds the tile kernels take, a request's tiles, attributes (call before any capture) */
bool ow_tile_supported(const MgWorldDesc &W);
long long ow_tiles(int nx, int nz);
/* whether the tiles do not take an area of more than `few` cells all the same: quart cells (qx0, qz0) to (qx1, qz1), `cells` of them
 * (or blocks in them) */
bool ow_beyond(bool fm, long long few, long long qx0, long long qz0, long long qx1, long long qz1, long long cells);
#define OT_FEW_CELLS 4096 /* for single grids and block maps */
#define OT_FEW_BLOCKS 1024
int ow_prepare();
/* records to provide for `cells` cells some of which are left to the exact evaluation (the double branch's with a target
 * open, well below 1 %; under the chunk-cell rule the tied ones too; cells beyond the record are evaluated in place) */
long long ow_open_cap(long long cells);
/* a group's requests (fm: the float branch's); open_pass: the recorded cells, after the tiles; overlap: the launch before this one
 * in the stream is a kernel of the same batch (overlap.cuh) */
int launch_ow_batch(bool fm, int tie, bool open_pass, bool overlap, const MgWorldDesc *d_worlds, const MgTreeNode *const *d_trees,
                    const MgBatchReq *d_reqs, int nreq, long long ntiles, const MgLattice *d_pool, unsigned long long *d_counter,
                    MgOpenCell *d_open, unsigned long long *d_nopen, long long open_cap, uint8_t *d_out, cudaStream_t st);

/* tile widths of the rest's four shapes for cells without a tile form (128 cells; the shapes differ in the register budget: 9, 7,
 * 6 and 8 resident CTAs per SM) */
extern const int kBatchTileWidths[BATCH_SHAPES];
/* tiles of a request of group `group`: 16 x 16 cells (owtile.cu); in the rest, 32 x 32 cells (nethertile.cuh), equal parts of up
 * to 24 x 24 chunks (endtile.cuh), or 128 quart cells of shape `shape` */
long long batch_tiles(int group, const MgWorldDesc &W, int qx0, int qz0, int nx, int nz, int shape);
/* lattices of a list of entries of one dimension; Overworld needs the prefix sums of lattices per entry; overlap: the launch before
 * this one in the stream is another dimension's */
int launch_setup_list(const MgWorldDesc *d_worlds, int dim, const MgSetupEntry *d_ent, int n, const int *d_first,
                      long long total_lattices, MgLattice *d_pool, bool overlap, cudaStream_t st);
/* kernel attributes and resident grid sizes; call before any stream capture */
int batch_prepare(int *ctas_per_sm);
/* d_reqs: the requests in group order, all under one tie rule.  ctas: upper bound on the rest's persistent grid, 0 = every
 * resident CTA of the shape.  d_counter: BATCH_COUNTERS counters.  d_open: open_cap[0] + open_cap[1] records for the open cells
 * of the double and the float group, finished by launches after the tiles (null: evaluated in place). */
int launch_batch(const MgWorldDesc *d_worlds, const MgTreeNode *const *d_trees, const MgBatchReq *d_reqs,
                 const BatchGroups &g, int tie, const MgLattice *d_pool, unsigned long long *d_counter, MgOpenCell *d_open,
                 const long long open_cap[2], uint8_t *d_out, int ctas, int shape, cudaStream_t st);
/* open_cap of a batch whose Overworld groups have `cells` cells */
void batch_open_cap(const long long cells[2], int tie, long long open_cap[2]);
}  // namespace mg
#endif
