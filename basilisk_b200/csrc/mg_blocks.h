/*
 * mg_blocks.h -- internal interface of the decomposed solve's kernels
 * (mg_blocks.cu): one launch works on every block of a device.  Plain C
 * types only.
 */
#ifndef MG_BLOCKS_H
#define MG_BLOCKS_H

#include "mg_launch.h"

#ifdef __cplusplus
extern "C" {
#endif

/* one block: its neighbours (block indices, -1: a box side, or the block's
   own periodic images), the conditions of a, and the finest level of a and b */
typedef struct {
  int nbr[6];
  int pad_[2];
  bmg_bcdesc bc;
  double * a;
  const double * b;
} bmg_blk;

/* one level of one block */
typedef struct {
  double * da, * da2, * res;
  bmg_coef alpha[3], lambda;
} bmg_blk_level;

/* the decomposition as the kernels see it, in device memory: nb blocks (of
   all devices), lv[level*nb + block], and the launch's own blocks mine[0..m) */
typedef struct {
  const bmg_blk * blk;
  const bmg_blk_level * lv;
  const int * mine;
  int nb, m;
} bmg_blocks;

/* a pass over level l (geometry g) of every block of the launch, with the
   boundary of da: the box images, and the images in the neighbours' ghost
   layers (peer memory when they live on another device).  mode RED / BLACK:
   in place; JACOBI: from da2 into da when odd, else from da into da2 */
int bmg_blocks_relax (int dim, int mode, int odd, bmg_geom g, int l, bmg_blocks B, double Delta,
                      cudaStream_t s);
/* zero (gc.n = 0) or bilinear prolongation of level l - 1 (whose iterate is
   in da2 when odd) into da of level l, with the same boundary */
int bmg_blocks_prolong (int dim, int odd, bmg_geom gc, bmg_geom g, int l, bmg_blocks B, cudaStream_t s);
/* two dimensions, l >= 1: nsweeps (at most BMG_BLOCKS_SWEEPS) red-black sweeps
   of level l from `in' (da, da2, zero, or the prolongation of level l - 1's
   da or da2) into `out' (da or da2; not `in'), with the images when images.
   No launch of the same sweeps on another device writes what it reads */
#define BMG_BLOCKS_SWEEPS 4
/* the cells of a level on a device up to which four sweeps of tiles beat
   eight passes: the window is three times the tile, which costs nothing
   while the passes are bound by their launches (2 x 2 blocks, ms per cycle
   with / without tiles on that level: 64^2 0.22 / 0.24, 128^2 0.23 / 0.25,
   256^2 0.34 / 0.35, 512^2 0.83 / 0.78, 1024^2 2.59 / 2.32) */
#define BMG_BLOCKS_TILE_CELLS (1 << 19)
enum { BMG_BLOCKS_DA = 0, BMG_BLOCKS_DA2, BMG_BLOCKS_COARSE_DA, BMG_BLOCKS_COARSE_DA2, BMG_BLOCKS_ZERO };
int bmg_blocks_tile (bmg_geom gc, bmg_geom g, int l, bmg_blocks B, const int * dims,
                     const int * periodic, double Delta, int in, int out, int nsweeps, int images,
                     cudaStream_t s);
/* restriction of res from level l + 1 into level l */
int bmg_blocks_restrict (int dim, bmg_geom gf, bmg_geom g, int l, bmg_blocks B, cudaStream_t s);
/* a += da (da2 when odd) on the finest level, with the boundary of a */
int bmg_blocks_correct (int dim, int odd, bmg_geom g, int l, bmg_blocks B, cudaStream_t s);
/* the residual of the finest level into res, max |res| over the launch's
   blocks into maxres */
int bmg_blocks_residual (int dim, bmg_geom g, int l, bmg_blocks B, double Delta,
                         unsigned long long * maxres, cudaStream_t s);
/* levels lo..hi of a cycle in one CTA, all blocks on its device: the
   restriction of res from level hi + 1 (when restrict_src), zero or
   prolongation and nrelax red-black sweeps of each level; dims, periodic:
   of the decomposition */
#define BMG_BLOCKS_CTA_CELLS 4096       /* cells of level hi, all blocks */
int bmg_blocks_bottom (int dim, const bmg_geom * g, const double * Delta, int lo, int hi,
                       bmg_blocks B, const int * dims, const int * periodic, int nrelax,
                       int restrict_src, cudaStream_t s);

#ifdef __cplusplus
}
#endif
#endif
