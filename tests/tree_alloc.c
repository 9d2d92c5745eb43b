/* Refining a quadtree when the device has no memory for the records of the
   shared-memory cycle, on a fake of the CUDA runtime: the tree is refined all
   the same, without them, and has them after the next refinement that finds
   the memory.  Exit status 0: so it was. */
#include "mg_tree_host.c"

/* the allocation that fails, counted from 1 (0: none) */
static int fail_at, count;
static void * given[1000];
const char * cudaGetErrorString (cudaError_t e) { (void) e; return "error"; }
cudaError_t cudaGetLastError (void) { return cudaSuccess; }
cudaError_t cudaSetDevice (int d) { (void) d; return cudaSuccess; }
cudaError_t cudaFree (void * p) { free (p); return cudaSuccess; }
cudaError_t cudaMalloc (void ** p, size_t n)
{
  *p = NULL;
  if (++count == fail_at) return cudaErrorMemoryAllocation;
  given[count] = *p = malloc (n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy (void * d, const void * s, size_t n, enum cudaMemcpyKind k)
{
  (void) k;
  if (!d || !s) return cudaErrorInvalidValue;
  memcpy (d, s, n);
  return cudaSuccess;
}
int bmg_i_fail (int status) { return status; }
int bmg_tree_interp_available (void) { return 1; }

static int corner (int level, double x, double y, double z, void * data)
{
  (void) z;
  return level < *(int *) data && x + y < 4./(1 << level);
}

int main (void)
{
  static bmg_grid g;
  g.dim = 2; g.depth = 6; g.L0 = 1.;
  size_t off = 0;
  for (int l = 0; l <= g.depth; l++) {
    const int n = 1 << l;
    g.g64[l].n = n; g.g64[l].xo = 8; g.g64[l].P = (n + 9 + 15)/16*16; g.g64[l].size = (long long) (n + 2)*g.g64[l].P;
    g.off64[l] = off;
    off += g.g64[l].size;
  }
  g.off64[g.depth + 1] = off;
  int depth = 5;
  if (bmg_tree_refine (&g, corner, &depth) <= 0 || g.tree->tc.slots <= 0) return 2;
  int records = 0;
  for (int k = 1; k <= count; k++) if (given[k] == g.tree->dtc) records = k;
  bmg_tree_free (&g);
  count = 0;
  fail_at = records;
  const int cells = bmg_tree_refine (&g, corner, &depth);
  if (cells <= 0 || !g.tree) { printf ("refining without memory for the records: %d\n", cells); return 4; }
  if (g.tree->tc.slots || g.tree->dtc) return 5;
  fail_at = 0;
  depth = 6;
  if (bmg_tree_refine (&g, corner, &depth) <= 0 || g.tree->tc.slots <= 0) return 6;
  bmg_tree_free (&g);
  return 0;
}
