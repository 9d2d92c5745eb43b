/* The decomposed solve's host code (mg_shard.c) on a fake of the CUDA runtime
   and of the launches, two blocks on two devices: the allocation of the
   second device's tables fails in one solve (argument 1) and succeeds in the
   next, which has to run with tables on both.  Exit status 0: it did. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "mg_grid.h"
#include "mg_blocks.h"

double TOLERANCE = 1e-3;
int NITERMAX = 100, NITERMIN = 1;

static int device, fail_at, mallocs, launches, bad;
static unsigned long long maxres;

#define OK { return cudaSuccess; }
cudaError_t cudaGetDevice (int * d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice (int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceCanAccessPeer (int * ok, int a, int b) { (void) a; (void) b; *ok = 1; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess (int d, unsigned f) { (void) d; (void) f; OK }
cudaError_t cudaStreamCreateWithFlags (cudaStream_t * s, unsigned f) { (void) f; *s = (cudaStream_t) 1; OK }
cudaError_t cudaStreamDestroy (cudaStream_t s) { (void) s; OK }
cudaError_t cudaStreamSynchronize (cudaStream_t s) { (void) s; OK }
cudaError_t cudaStreamWaitEvent (cudaStream_t s, cudaEvent_t e, unsigned f) { (void) s; (void) e; (void) f; OK }
cudaError_t cudaEventCreateWithFlags (cudaEvent_t * e, unsigned f) { (void) f; *e = (cudaEvent_t) 1; OK }
cudaError_t cudaEventDestroy (cudaEvent_t e) { (void) e; OK }
cudaError_t cudaEventRecord (cudaEvent_t e, cudaStream_t s) { (void) e; (void) s; OK }
cudaError_t cudaEventElapsedTime (float * t, cudaEvent_t a, cudaEvent_t b) { (void) a; (void) b; *t = 0.f; OK }
cudaError_t cudaGetLastError (void) OK
const char * cudaGetErrorString (cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaFree (void * p) { free (p); OK }

cudaError_t cudaMalloc (void ** p, size_t n)
{
  *p = NULL;
  if (++mallocs == fail_at) return cudaErrorMemoryAllocation;
  *p = malloc (n);
  return cudaSuccess;
}

cudaError_t cudaMemcpyAsync (void * d, const void * s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
  (void) k; (void) st;
  if (!d || !s) return cudaErrorInvalidValue;
  memcpy (d, s, n);
  return cudaSuccess;
}

cudaError_t cudaMemsetAsync (void * d, int v, size_t n, cudaStream_t st) { (void) st; memset (d, v, n); OK }

static int launched (bmg_blocks B) { launches++; if (!B.blk || !B.lv || !B.mine) bad++; return 0; }
int bmg_blocks_relax (int dim, int mode, int odd, bmg_geom g, int l, bmg_blocks B, double D, cudaStream_t s)
{ (void) dim; (void) mode; (void) odd; (void) g; (void) l; (void) D; (void) s; return launched (B); }
int bmg_blocks_prolong (int dim, int odd, bmg_geom gc, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{ (void) dim; (void) odd; (void) gc; (void) g; (void) l; (void) s; return launched (B); }
int bmg_blocks_tile (bmg_geom gc, bmg_geom g, int l, bmg_blocks B, const int * dims, const int * periodic,
                     double D, int in, int out, int ns, int images, cudaStream_t s)
{ (void) gc; (void) g; (void) l; (void) dims; (void) periodic; (void) D; (void) in; (void) out; (void) ns;
  (void) images; (void) s; return launched (B); }
int bmg_blocks_restrict (int dim, bmg_geom gf, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{ (void) dim; (void) gf; (void) g; (void) l; (void) s; return launched (B); }
int bmg_blocks_correct (int dim, int odd, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{ (void) dim; (void) odd; (void) g; (void) l; (void) s; return launched (B); }
int bmg_blocks_residual (int dim, bmg_geom g, int l, bmg_blocks B, double D, unsigned long long * m, cudaStream_t s)
{ (void) dim; (void) g; (void) l; (void) D; (void) m; (void) s; return launched (B); }
int bmg_blocks_bottom (int dim, const bmg_geom * g, const double * D, int lo, int hi, bmg_blocks B,
                       const int * dims, const int * periodic, int nrelax, int src, cudaStream_t s)
{ (void) dim; (void) g; (void) D; (void) lo; (void) hi; (void) dims; (void) periodic; (void) nrelax; (void) src;
  (void) s; return launched (B); }
int bmg_launch_halo (int dim, bmg_geom g, int e, const bmg_halo * b, int nb, cudaStream_t s)
{ (void) dim; (void) g; (void) e; (void) b; (void) nb; (void) s; return 0; }
int bmg_launch_relax (int dim, int st, int mode, bmg_geom g, void * o, const void * i, const void * r,
                      const bmg_coef * a, bmg_coef l, double D, const bmg_bcdesc * bc, cudaStream_t s)
{ (void) dim; (void) st; (void) mode; (void) g; (void) o; (void) i; (void) r; (void) a; (void) l; (void) D;
  (void) bc; (void) s; return 0; }
int bmg_launch_restrict (int dim, int sf, int sc, bmg_geom gf, bmg_geom gc, const void * f, void * c, cudaStream_t s)
{ (void) dim; (void) sf; (void) sc; (void) gf; (void) gc; (void) f; (void) c; (void) s; return 0; }
int bmg_launch_restrict_face (int dim, bmg_geom gf, bmg_geom gc, const double * const * f, double * const * c,
                              int p, cudaStream_t s)
{ (void) dim; (void) gf; (void) gc; (void) f; (void) c; (void) p; (void) s; return 0; }
int bmg_launch_sum (int dim, bmg_geom g, const double * b, double * p, int n, double * o, cudaStream_t s)
{ (void) dim; (void) g; (void) b; (void) p; (void) n; (void) o; (void) s; return 0; }

static double values[3][64];
static field_t fields[3];
int bmg_i_fail (int status) { return status; }
field_t * bmg_i_field (bmg_grid * g, int h) { (void) g; return h > 0 && h < 3 ? &fields[h] : NULL; }
void bmg_i_bcdesc (const bmg_grid * g, const field_t * f, bmg_bcdesc * bc) { (void) g; (void) f; memset (bc, 0, sizeof *bc); }
int bmg_i_workspace (bmg_grid * g) { (void) g; return 0; }
double * bmg_i_ws64 (bmg_grid * g, int which, int l) { (void) g; (void) which; (void) l; return values[0]; }
int bmg_set_stream (bmg_grid * g, void * s) { (void) g; (void) s; return 0; }

int main (int argc, char ** argv)
{
  static bmg_grid grids[2];
  static double pinned[2][4], sum;
  bmg_grid * blocks[2];
  for (int b = 0; b < 2; b++) {
    grids[b].dim = 1; grids[b].depth = 2; grids[b].device = b; grids[b].L0 = 1.;
    grids[b].relax = BMG_RELAX_RBGS; grids[b].precision = BMG_FP64;
    grids[b].h_pinned = pinned[b]; grids[b].d_maxres = &maxres; grids[b].d_sum = &sum;
    for (int l = 0; l <= 2; l++) { grids[b].g64[l].n = 1 << l; grids[b].g64[l].size = 8; }
    blocks[b] = &grids[b];
  }
  for (int f = 1; f < 3; f++) {
    fields[f].used = 1; fields[f].face_dim = -1;
    for (int l = 0; l <= 2; l++) fields[f].lv[l] = values[f];
  }
  const int dims[3] = {2, 1, 1};
  bmg_shard * s = NULL;
  if (bmg_shard_new (&s, blocks, dims, NULL)) return 2;
  struct Poisson p;
  memset (&p, 0, sizeof p);
  p.a.i = 1; p.b.i = 2;
  mgstats st;
  fail_at = argc > 1 ? atoi (argv[1]) : 2;
  if (bmg_shard_poisson (s, p, &st) != BMG_ENOMEM) return 3;
  if (launches) return 4;                       /* nothing ran without its tables */
  const int r = bmg_shard_poisson (s, p, &st);
  if (r != BMG_OK) { printf ("the solve after a failed allocation: status %d\n", r); return 5; }
  if (!launches || bad) return 6;
  const int before = mallocs;
  if (bmg_shard_poisson (s, p, &st) != BMG_OK || mallocs != before) return 7;
  bmg_shard_free (s);
  return 0;
}
