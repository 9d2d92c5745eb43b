/*
 * mg_blocks.cu -- kernels of the solve over a domain decomposed into blocks
 * (mg_shard.c, the counterpart of grid/multigrid-mpi.h), FP64, 1D to 3D.
 *
 * Every launch works on all the blocks of its device, and the thread that
 * writes a cell writes all its images: the box ghosts of its own block, and
 * the ghost cells of the neighbouring blocks that mirror it (edges and
 * corners included), in the neighbour's array -- peer memory over NVLink
 * when the neighbour lives on another device.  A pass is then one launch
 * per device with no exchange after it, where it took a launch per block
 * and one per direction.  No launch reads what it or a launch on another
 * device writes at the same time: a colour pass reads the other colour only
 * (n is even, so an image in a neighbour keeps its colour), a Jacobi sweep
 * and a prolongation write another array than they read, the correction
 * reads interior cells only.
 *
 * The images are those of the exchange they replace (slabs direction by
 * direction, ghosts of the earlier directions included): the product over
 * the directions of a cell's own position, its box ghost, its periodic image
 * in the block, or its image in the neighbour, with the owner's conditions.
 * Cell updates are relax_value's, k_prolong's, k_restrict's and k_residual's
 * expressions in their order: bit-identical to one grid over the domain.
 */
#include <cuda_runtime.h>
#include <string.h>
#include "mg_device.cuh"
#include "mg_blocks.h"

using namespace bmgd;

namespace {

/* cell q of level l (n = 2^l) in C order */
template <int DIM>
__device__ __forceinline__ void cell_at (long long q, int l, int & i, int & j, int & k)
{
  const int m = (1 << l) - 1;
  if (DIM == 1) { i = (int) q; j = k = 0; }
  else if (DIM == 2) { i = (int) (q >> l); j = (int) q & m; k = 0; }
  else { i = (int) (q >> (2*l)); j = (int) (q >> l) & m; k = (int) q & m; }
}

/* write every image of cell (i, j, k) of block b, value v: f (t) is the
   array of block t that the launch writes, hom the homogeneous conditions
   (of da) or not (of a) */
template <int DIM, typename F>
__device__ __noinline__ void images (const bmg_blk * B, int b, const bmg_geom & g, int i, int j, int k,
                                     double v, bool hom, F f)
{
  const int n = g.n, c[3] = {i, j, k};
  const bmg_bcdesc & bc = B[b].bc;
  /* level 0 of a block with periodic directions of its own: every neighbour
     of the single cell is a copy of it (multigrid.h:655-664) */
  const bool copies = n == 1 && (bc.periodic[0] || bc.periodic[1] || bc.periodic[2]);
  /* per direction: the cell itself, and up to two images, each a position
     and a side s: the box ghost of side s (kind 1), the neighbour on side s
     (kind 2), or the block's own periodic image (kind 0) */
  int pos[3][3], sd[3][3], kind[3][3], cnt[3];
  for (int e = 0; e < 3; e++) {
    pos[e][0] = c[e]; sd[e][0] = -1; kind[e][0] = 0; cnt[e] = 1;
    if (e < DIM)
      for (int hi = 0; hi < 2; hi++)
        if (c[e] == (hi ? n - 1 : 0)) {
          const int s = 2*e + (hi ? 0 : 1), t = B[b].nbr[s], q = cnt[e]++;
          sd[e][q] = s;
          kind[e][q] = t >= 0 ? 2 : bc.periodic[e] ? 0 : 1;
          /* beyond the side for a box ghost, across for an image */
          pos[e][q] = (kind[e][q] == 1) == (hi == 1) ? n : -1;
        }
  }
  for (int x = 0; x < cnt[0]; x++)
    for (int y = 0; y < cnt[1]; y++)
      for (int z = 0; z < cnt[2]; z++) {
        if (x == 0 && y == 0 && z == 0) continue;
        const int at[3] = {x, y, z};
        double r = v;
        int t = b;
        for (int e = 0; e < DIM; e++) {
          const int q = at[e], s = sd[e][q];
          if (kind[e][q] == 2) t = B[t].nbr[s];
          else if (kind[e][q] == 1 && !copies) {
            if (hom) r = bc.type[s] == 1 /* BMG_DIRICHLET */ ? r*(-1.) : r;
            else {
              const double w = bc_data<DIM> (bc, s, n, i, j, k);
              r = bc.type[s] == 1 ? 2.*(w) - r : bc.Delta*(w) + r;
            }
          }
        }
        f (t)[cidx<DIM> (g, pos[0][x], pos[1][y], pos[2][z])] = r;
      }
}

template <int DIM, typename F>
__device__ __forceinline__ void put (const bmg_blk * B, int b, const bmg_geom & g, int i, int j, int k,
                                     double v, bool hom, F f)
{
  f (b)[cidx<DIM> (g, i, j, k)] = v;
  if (on_boundary<DIM> (g.n, i, j, k)) images<DIM> (B, b, g, i, j, k, v, hom, f);
}

/* the update of one cell of block b of level l */
template <int DIM>
__device__ __forceinline__ double update (const bmg_blk_level & L, const bmg_geom & g, long long id,
                                          const double * in, double D2)
{
  return relax_value<DIM, double> (g, id, in, L.res, coef_of<double> (L.alpha[0]),
                                   coef_of<double> (L.alpha[1]), coef_of<double> (L.alpha[2]),
                                   coef_of<double> (L.lambda), D2);
}

/* cell h of the n/2 of one colour in a row */
template <int DIM>
__device__ __forceinline__ void colour_cell (long long q, int l, int colour, int & i, int & j, int & k)
{
  const int lh = l - 1, m = (1 << l) - 1, h = (int) q & ((1 << lh) - 1);
  const long long row = q >> lh;
  if (DIM == 1) { i = 2*h + colour; j = k = 0; }
  else if (DIM == 2) { i = (int) row; j = 2*h + ((colour + i) & 1); k = 0; }
  else { i = (int) (row >> l); j = (int) row & m; k = 2*h + ((colour + i + j) & 1); }
}

/* blockIdx.y: the block (of the launch's own); a thread per cell of the
   colour, or per cell (Jacobi) */
template <int DIM, int MODE>
__global__ void k_blocks_relax (bmg_geom g, int l, bmg_blocks B, double Delta, int odd)
{
  pdl_wait ();
  pdl_trigger ();
  const long long q = (long long) blockIdx.x*blockDim.x + threadIdx.x;
  const long long cells = 1LL << (DIM*l);
  if (q >= (MODE == BMG_SWEEP_JACOBI ? cells : cells/2)) return;
  const int b = B.mine[blockIdx.y];
  const bmg_blk_level * lv = B.lv + (long long) l*B.nb;
  const bmg_blk_level & L = lv[b];
  int i, j, k;
  if (MODE == BMG_SWEEP_JACOBI) cell_at<DIM> (q, l, i, j, k);
  else colour_cell<DIM> (q, l, MODE == BMG_SWEEP_RED ? 0 : 1, i, j, k);
  const long long id = cidx<DIM> (g, i, j, k);
  if (MODE == BMG_SWEEP_JACOBI) {
    const double * in = odd ? L.da2 : L.da;
    const double c = update<DIM> (L, g, id, in, Delta*Delta);
    put<DIM> (B.blk, b, g, i, j, k, (in[id] + 2.*c)/3., true,
              [=] (int t) { return odd ? lv[t].da : lv[t].da2; });
  }
  else
    put<DIM> (B.blk, b, g, i, j, k, update<DIM> (L, g, id, L.da, Delta*Delta), true,
              [=] (int t) { return lv[t].da; });
}

/* bilinear (multigrid-common.h:124-140) in k_prolong's expression and order */
template <int DIM>
__device__ __forceinline__ double bilinear (const bmg_geom & gc, const double * s, int i, int j, int k)
{
  const int pi = i >> 1, cx = (i & 1) ? 1 : -1, pj = j >> 1, cy = (j & 1) ? 1 : -1;
  if (DIM == 1)
    return (3.*s[cidx<1> (gc, pi, 0, 0)] + s[cidx<1> (gc, pi + cx, 0, 0)])/4.;
  if (DIM == 2)
    return (9.*s[cidx<2> (gc, pi, pj, 0)] +
            3.*(s[cidx<2> (gc, pi + cx, pj, 0)] + s[cidx<2> (gc, pi, pj + cy, 0)]) +
            s[cidx<2> (gc, pi + cx, pj + cy, 0)])/16.;
  const int pk = k >> 1, cz = (k & 1) ? 1 : -1;
  return (27.*s[cidx<3> (gc, pi, pj, pk)] +
          9.*(s[cidx<3> (gc, pi + cx, pj, pk)] + s[cidx<3> (gc, pi, pj + cy, pk)] +
              s[cidx<3> (gc, pi, pj, pk + cz)]) +
          3.*(s[cidx<3> (gc, pi + cx, pj + cy, pk)] + s[cidx<3> (gc, pi + cx, pj, pk + cz)] +
              s[cidx<3> (gc, pi, pj + cy, pk + cz)]) +
          s[cidx<3> (gc, pi + cx, pj + cy, pk + cz)])/64.;
}

template <int DIM>
__global__ void k_blocks_prolong (bmg_geom gc, bmg_geom g, int l, bmg_blocks B, int odd)
{
  pdl_wait ();
  pdl_trigger ();
  const long long q = (long long) blockIdx.x*blockDim.x + threadIdx.x;
  if (q >= 1LL << (DIM*l)) return;
  const int b = B.mine[blockIdx.y];
  const bmg_blk_level * lv = B.lv + (long long) l*B.nb;
  int i, j, k;
  cell_at<DIM> (q, l, i, j, k);
  double v = 0.;
  if (gc.n) {
    const bmg_blk_level & C = (lv - B.nb)[b];
    v = bilinear<DIM> (gc, odd ? C.da2 : C.da, i, j, k);
  }
  put<DIM> (B.blk, b, g, i, j, k, v, true, [=] (int t) { return lv[t].da; });
}

/* restriction_average (multigrid-common.h:26-32) in foreach_child order */
template <int DIM>
__device__ __forceinline__ double mean (const bmg_geom & gf, const double * f, int i, int j, int k)
{
  double sum = 0.;
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < (DIM > 1 ? 2 : 1); b++)
#pragma unroll
      for (int d = 0; d < (DIM > 2 ? 2 : 1); d++)
        sum += f[cidx<DIM> (gf, 2*i + a, 2*j + b, 2*k + d)];
  return sum/(double) (1 << DIM);
}

template <int DIM>
__global__ void k_blocks_restrict (bmg_geom gf, bmg_geom g, int l, bmg_blocks B)
{
  pdl_wait ();
  pdl_trigger ();
  const long long q = (long long) blockIdx.x*blockDim.x + threadIdx.x;
  if (q >= 1LL << (DIM*l)) return;
  const bmg_blk_level * lv = B.lv + (long long) l*B.nb + B.mine[blockIdx.y];
  int i, j, k;
  cell_at<DIM> (q, l, i, j, k);
  lv->res[cidx<DIM> (g, i, j, k)] = mean<DIM> (gf, lv[B.nb].res, i, j, k);
}

template <int DIM>
__global__ void k_blocks_correct (bmg_geom g, int l, bmg_blocks B, int odd)
{
  pdl_wait ();
  pdl_trigger ();
  const long long q = (long long) blockIdx.x*blockDim.x + threadIdx.x;
  if (q >= 1LL << (DIM*l)) return;
  const int b = B.mine[blockIdx.y];
  const bmg_blk_level & L = B.lv[(long long) l*B.nb + b];
  int i, j, k;
  cell_at<DIM> (q, l, i, j, k);
  const long long id = cidx<DIM> (g, i, j, k);
  const bmg_blk * blk = B.blk;
  put<DIM> (blk, b, g, i, j, k, blk[b].a[id] + (odd ? L.da2 : L.da)[id], false,
            [=] (int t) { return blk[t].a; });
}

/* k_residual's expression and order (poisson.h:373-389) */
template <int DIM, bool POW2>
__global__ void k_blocks_residual (bmg_geom g, int l, bmg_blocks B, double Delta,
                                   unsigned long long * maxres)
{
  pdl_wait ();
  pdl_trigger ();
  const long long q = (long long) blockIdx.x*blockDim.x + threadIdx.x;
  double m = 0.;
  const double rD = 1./Delta;
  if (q < 1LL << (DIM*l)) {
    const int b = B.mine[blockIdx.y];
    const bmg_blk_level & L = B.lv[(long long) l*B.nb + b];
    int i, j, k;
    cell_at<DIM> (q, l, i, j, k);
    const long long id = cidx<DIM> (g, i, j, k);
    const double * a = B.blk[b].a, ac = a[id];
    const Coef<double> lam = coef_of<double> (L.lambda);
    double r = B.blk[b].b[id] - lam.at (id)*ac;
#pragma unroll
    for (int e = 0; e < DIM; e++) {
      const Coef<double> al = coef_of<double> (L.alpha[e]);
      const long long s = cstride<DIM> (g, e);
      r += over_delta<POW2> (al.at (id)*over_delta<POW2> (ac - a[id - s], Delta, rD) -
                             al.at (id + s)*over_delta<POW2> (a[id + s] - ac, Delta, rD), Delta, rD);
    }
    L.res[id] = r;
    m = fabs (r);
  }
  block_max_atomic (m, maxres);
}

struct BottomParams {
  bmg_geom g[BMG_MAXLEVEL + 1];
  double Delta[BMG_MAXLEVEL + 1];
  bmg_blocks B;
  int lo, hi, nrelax, restrict_src;
};

/* the coarse levels of all the blocks in one CTA: a barrier between passes
   instead of a launch (its own global writes are visible to the CTA after
   the barrier, and its L1 serves them).  Bound: the latency of a pass.  For
   the levels that k_blocks_staged cannot hold. */
template <int DIM>
__global__ void __launch_bounds__ (1024, 1) k_blocks_bottom (const __grid_constant__ BottomParams P)
{
  pdl_wait ();
  pdl_trigger ();
  const bmg_blocks & B = P.B;
  for (int l = P.restrict_src ? P.hi : P.hi - 1; l >= P.lo; l--) {
    const int cells = 1 << (DIM*l);
    for (int q = threadIdx.x; q < cells*B.m; q += blockDim.x) {
      const bmg_blk_level * lv = B.lv + (long long) l*B.nb + B.mine[q >> (DIM*l)];
      int i, j, k;
      cell_at<DIM> (q & (cells - 1), l, i, j, k);
      lv->res[cidx<DIM> (P.g[l], i, j, k)] = mean<DIM> (P.g[l + 1], lv[B.nb].res, i, j, k);
    }
    __syncthreads ();
  }
  for (int l = P.lo; l <= P.hi; l++) {
    const bmg_geom & g = P.g[l];
    const bmg_blk_level * lv = B.lv + (long long) l*B.nb;
    const int cells = 1 << (DIM*l);
    auto da = [=] (int t) { return lv[t].da; };
    for (int q = threadIdx.x; q < cells*B.m; q += blockDim.x) {
      const int b = B.mine[q >> (DIM*l)];
      int i, j, k;
      cell_at<DIM> (q & (cells - 1), l, i, j, k);
      const double v = l == P.lo ? 0. : bilinear<DIM> (P.g[l - 1], (lv - B.nb)[b].da, i, j, k);
      put<DIM> (B.blk, b, g, i, j, k, v, true, da);
    }
    __syncthreads ();
    const double D2 = P.Delta[l]*P.Delta[l];
    for (int p = 0; p < 2*P.nrelax; p++) {
      for (int q = threadIdx.x; q < (cells >> 1)*B.m; q += blockDim.x) {
        const int b = B.mine[q >> (DIM*l - 1)];
        int i, j, k;
        colour_cell<DIM> (q & ((cells >> 1) - 1), l, p & 1, i, j, k);
        const long long id = cidx<DIM> (g, i, j, k);
        put<DIM> (B.blk, b, g, i, j, k, update<DIM> (lv[b], g, id, lv[b].da, D2), true, da);
      }
      __syncthreads ();
    }
  }
}

/* ---------------------------------------------------------------- */
/* the same levels as one grid in shared memory                      */
/* ---------------------------------------------------------------- */

#define ST_THREADS 1024
/* the shared memory of one CTA */
#define ST_BYTES (227*1024)

struct StagedParams {
  BottomParams bot;
  int dims[3], periodic[3];       /* of the decomposition */
  unsigned off_c, off_w, off_nb;  /* shared memory: coarser iterate, weights, neighbours */
};

/* a level of the blocks as one grid, its cells split by colour: extents,
   half the cells, half a row */
template <int DIM>
struct Joint {
  int l, N[3], half, nh;
  __device__ __forceinline__ Joint (const StagedParams & P, int level) : l (level)
  {
    half = 1;
#pragma unroll
    for (int e = 0; e < 3; e++) { N[e] = e < DIM ? P.dims[e] << l : 1; half *= N[e]; }
    half >>= 1;
    nh = N[DIM - 1] >> 1;
  }
  __device__ __forceinline__ int slot (const int * x) const
  {
    const int row = DIM == 1 ? 0 : DIM == 2 ? x[0] : x[0]*N[1] + x[1];
    const int c = (x[0] + (DIM > 1 ? x[1] : 0) + (DIM > 2 ? x[2] : 0)) & 1;
    return c*half + row*nh + (x[DIM - 1] >> 1);
  }
  /* cell q of colour c */
  __device__ __forceinline__ void cell (int c, int q, int * x) const
  {
    const int row = q/nh, h = q - row*nh;
    x[0] = x[1] = x[2] = 0;
    if (DIM == 2) x[0] = row;
    if (DIM == 3) { x[0] = row/N[1]; x[1] = row - x[0]*N[1]; }
    x[DIM - 1] = 2*h + ((c + x[0] + x[1]) & 1);
  }
  __device__ __forceinline__ int block (const StagedParams & P, const int * x) const
  {
    return ((x[0] >> l)*P.dims[1] + (DIM > 1 ? x[1] >> l : 0))*P.dims[2] + (DIM > 2 ? x[2] >> l : 0);
  }
  /* iterate u at a cell, or at a position beyond the sides: the image of
     the cell it mirrors, with its block's conditions */
  __device__ __forceinline__ double at (const StagedParams & P, const double * u, int i, int j, int k) const
  {
    int x[3] = {i, j, k}, side[3];
    bool box = false;
#pragma unroll
    for (int e = 0; e < DIM; e++) {
      side[e] = -1;
      if (x[e] >= 0 && x[e] < N[e]) continue;
      const bool lo = x[e] < 0;
      if (P.periodic[e]) x[e] = lo ? N[e] - 1 : 0;
      else { x[e] = lo ? 0 : N[e] - 1; side[e] = 2*e + lo; box = true; }
    }
    double v = u[slot (x)];
    if (box) {
      const bmg_bcdesc & bc = P.bot.B.blk[block (P, x)].bc;
#pragma unroll
      for (int e = 0; e < DIM; e++)
        if (side[e] >= 0 && bc.type[side[e]] == 1 /* BMG_DIRICHLET */) v = v*(-1.);
    }
    return v;
  }
};

/* the prolongation of level l - 1 (k_prolong's expression and order) at a
   cell of level l */
template <int DIM>
__device__ __forceinline__ double staged_bilinear (const StagedParams & P, const Joint<DIM> & C,
                                                   const double * s, const int * x)
{
  const int pi = x[0] >> 1, cx = (x[0] & 1) ? 1 : -1, pj = x[1] >> 1, cy = (x[1] & 1) ? 1 : -1;
  const int pk = x[2] >> 1, cz = (x[2] & 1) ? 1 : -1;
  auto a = [&] (int i, int j, int k) { return C.at (P, s, i, j, k); };
  if (DIM == 1) return (3.*a (pi, 0, 0) + a (pi + cx, 0, 0))/4.;
  if (DIM == 2)
    return (9.*a (pi, pj, 0) + 3.*(a (pi + cx, pj, 0) + a (pi, pj + cy, 0)) + a (pi + cx, pj + cy, 0))/16.;
  return (27.*a (pi, pj, pk) + 9.*(a (pi + cx, pj, pk) + a (pi, pj + cy, pk) + a (pi, pj, pk + cz)) +
          3.*(a (pi + cx, pj + cy, pk) + a (pi + cx, pj, pk + cz) + a (pi, pj + cy, pk + cz)) +
          a (pi + cx, pj + cy, pk + cz))/64.;
}

/* zero or prolongation, then the sweeps of one level: u its iterate, c that
   of the level below.  A thread owns NS cells of each colour.  The image of
   a box side is read only by the cell it mirrors, whose weight takes its
   sign and whose neighbour there is the cell itself.  Weights and
   neighbours stay in registers when NS = 1, in shared memory (the thread's
   own words) otherwise. */
template <int DIM, int NS>
__device__ __noinline__ void staged_level (const StagedParams & P, int l)
{
  extern __shared__ __align__ (16) unsigned char ssm[];
  const bool even = (P.bot.hi - l) & 1;
  double * u = (double *) (ssm + (even ? P.off_c : 0));
  const double * uc = (const double *) (ssm + (even ? 0 : P.off_c));
  double * W = (double *) (ssm + P.off_w);
  ushort2 * NB = (ushort2 *) (ssm + P.off_nb);
  const Joint<DIM> G (P, l), C (P, l > 0 ? l - 1 : 0);
  const int tid = threadIdx.x, half = G.half, cells = 2*half;
  const int active = half < ST_THREADS ? (half + 31) & ~31 : ST_THREADS;
  const double D2 = P.bot.Delta[l]*P.bot.Delta[l];
  double w[2][2*DIM], be[2][NS], d[2][NS], y[2][NS];
  int nb[2][2*DIM];
  bool plain = false;             /* a diagonal outside exact_quotient's range */
#pragma unroll
  for (int c = 0; c < 2; c++)
#pragma unroll
    for (int s = 0; s < NS; s++) {
      const int q = tid + s*ST_THREADS;
      if (q >= half) continue;
      int x[3];
      G.cell (c, q, x);
      const int b = G.block (P, x), p = c*half + q, m = (1 << l) - 1;
      const bmg_blk_level & L = P.bot.B.lv[(long long) l*P.bot.B.nb + b];
      const bmg_geom & g = P.bot.g[l];
      const long long id = cidx<DIM> (g, x[0] & m, x[1] & m, x[2] & m);
      be[c][s] = (-D2)*L.res[id];
      double dd = (-coef_of<double> (L.lambda).at (id))*D2;
#pragma unroll
      for (int e = 0; e < DIM; e++) {
        const Coef<double> al = coef_of<double> (L.alpha[e]);
        const double w1 = al.at (id + cstride<DIM> (g, e)), w0 = al.at (id);
        dd += w1 + w0;
        double wv[2];
        int at[2];
#pragma unroll
        for (int lo = 0; lo < 2; lo++) {
          const bool edge = x[e] == (lo ? 0 : G.N[e] - 1), box = edge && !P.periodic[e];
          const double v = lo ? w0 : w1;
          wv[lo] = box && P.bot.B.blk[b].bc.type[2*e + lo] == 1 ? -v : v;
          int z[3] = {x[0], x[1], x[2]};
          z[e] = edge ? (lo ? G.N[e] - 1 : 0) : x[e] + (lo ? -1 : 1);
          at[lo] = box ? p : G.slot (z);
        }
        if (NS == 1) {
          w[c][2*e] = wv[0]; w[c][2*e + 1] = wv[1];
          nb[c][2*e] = at[0]; nb[c][2*e + 1] = at[1];
        }
        else {
          W[2*e*cells + p] = wv[0]; W[(2*e + 1)*cells + p] = wv[1];
          NB[e*cells + p] = make_ushort2 (at[0], at[1]);
        }
      }
      d[c][s] = dd;
      y[c][s] = 1./dd;
      plain = plain || divisor_unsafe (dd);
      u[p] = l == P.bot.lo ? 0. : staged_bilinear<DIM> (P, C, uc, x);
    }
  __syncthreads ();
  if (tid < active)
    for (int sw = 0; sw < P.bot.nrelax; sw++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
#pragma unroll
        for (int s = 0; s < NS; s++) {
          const int q = tid + s*ST_THREADS, p = c*half + q;
          if (q >= half) continue;
          double m = be[c][s];
#pragma unroll
          for (int e = 0; e < DIM; e++)
            if (NS == 1) m = m + (w[c][2*e]*u[nb[c][2*e]] + w[c][2*e + 1]*u[nb[c][2*e + 1]]);
            else {
              const ushort2 at = NB[e*cells + p];
              m = m + (W[2*e*cells + p]*u[at.x] + W[(2*e + 1)*cells + p]*u[at.y]);
            }
          double v = exact_quotient (m, d[c][s], y[c][s]);
          if (__any_sync (__activemask (), plain || quotient_unsafe (m))) v = m/d[c][s];
          u[p] = v;
        }
        asm volatile ("bar.sync 1, %0;" :: "r" (active) : "memory");
      }
  __syncthreads ();
}

/* k_blocks_bottom's levels with the blocks joined into one grid (they are
   one: a block's ghosts are its neighbours' cells): the iterate split by
   colour in shared memory, one copy of a cell instead of its images, the
   coefficients read once per level, quotients through the diagonal's
   reciprocal.  Only level hi's iterate goes back to the blocks, with all
   its images.  The residual is restricted in the blocks' arrays.  Bound:
   the latency of a pass, and at 4096 cells its shared-memory accesses.
   2 x 2 blocks of 128^2, levels of 4 to 4096 cells: 249 us per cycle as
   passes over global memory (k_blocks_bottom), 100 us here. */
template <int DIM>
__global__ void __launch_bounds__ (ST_THREADS, 1) k_blocks_staged (const __grid_constant__ StagedParams P)
{
  extern __shared__ __align__ (16) unsigned char ssm[];
  pdl_wait ();
  pdl_trigger ();
  const bmg_blocks & B = P.bot.B;
  for (int l = P.bot.restrict_src ? P.bot.hi : P.bot.hi - 1; l >= P.bot.lo; l--) {
    const int cells = 1 << (DIM*l);
    for (int q = threadIdx.x; q < cells*B.m; q += blockDim.x) {
      const bmg_blk_level * lv = B.lv + (long long) l*B.nb + (q >> (DIM*l));
      int i, j, k;
      cell_at<DIM> (q & (cells - 1), l, i, j, k);
      lv->res[cidx<DIM> (P.bot.g[l], i, j, k)] = mean<DIM> (P.bot.g[l + 1], lv[B.nb].res, i, j, k);
    }
    __syncthreads ();
  }
  for (int l = P.bot.lo; l <= P.bot.hi; l++)
    if (Joint<DIM> (P, l).half <= ST_THREADS) staged_level<DIM, 1> (P, l);
    else staged_level<DIM, 2> (P, l);
  const int l = P.bot.hi, n = 1 << l, e = n + 2, cells = DIM == 1 ? e : DIM == 2 ? e*e : e*e*e;
  const Joint<DIM> G (P, l);
  const double * u = (const double *) ssm;
  for (int q = threadIdx.x; q < cells*B.m; q += blockDim.x) {
    const int b = q/cells, r = q - b*cells;
    const int i = (DIM == 1 ? r : DIM == 2 ? r/e : r/(e*e)) - 1;
    const int j = DIM == 1 ? 0 : (DIM == 2 ? r % e : r/e % e) - 1, k = DIM == 3 ? r % e - 1 : 0;
    const int b0 = b/(P.dims[1]*P.dims[2]), b1 = b/P.dims[2] % P.dims[1], b2 = b % P.dims[2];
    B.lv[(long long) l*B.nb + b].da[cidx<DIM> (P.bot.g[l], i, j, k)] =
      G.at (P, u, (b0 << l) + i, (b1 << l) + j, (b2 << l) + k);
  }
}

int status_of (cudaError_t launched)
{
  const cudaError_t e = cudaGetLastError ();
  return launched != cudaSuccess ? (int) launched : (int) e;
}

/* the launch, or -1 when the levels don't fit the shared memory (three
   dimensions above some 3300 cells) */
template <int DIM>
int staged_dim (const BottomParams & bot, const int * dims, const int * periodic, cudaStream_t s)
{
  long long cells = (long long) bot.B.nb << (DIM*bot.hi);
  if (bot.B.m != bot.B.nb || cells > 4*ST_THREADS) return -1;
  StagedParams P;
  memset (&P, 0, sizeof P);
  P.bot = bot;
  for (int e = 0; e < 3; e++) { P.dims[e] = e < DIM ? dims[e] : 1; P.periodic[e] = e < DIM && periodic[e]; }
  const bool words = cells > 2*ST_THREADS;
  P.off_c = (unsigned) (cells*8);
  P.off_w = P.off_c + (unsigned) (cells*8 >> DIM);
  P.off_nb = P.off_w + (words ? (unsigned) (cells*2*DIM*8) : 0);
  const unsigned bytes = P.off_nb + (words ? (unsigned) (cells*DIM*sizeof (ushort2)) : 0);
  if (bytes > ST_BYTES) return -1;
  static unsigned char configured[64];
  int dev = 0;
  cudaGetDevice (&dev);
  if (dev < 0 || dev >= 64) return (int) cudaErrorInvalidDevice;
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute (k_blocks_staged<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_BYTES);
    if (e != cudaSuccess) return (int) e;
    configured[dev] = 1;
  }
  return status_of (pdl_launch (k_blocks_staged<DIM>, dim3 (1), dim3 (ST_THREADS), bytes, s, P));
}

/* ---------------------------------------------------------------- */
/* several sweeps per launch, two dimensions                         */
/* ---------------------------------------------------------------- */

/* cells of a tile, its sweeps, and the cells around it that they need */
#define BT_I 32
#define BT_J 16
#define BT_HALO (2*BMG_BLOCKS_SWEEPS)
#define BT_THREADS ((BT_I + 2*BT_HALO)*(BT_J + 2*BT_HALO)/2)

struct TileParams {
  bmg_geom gc, g;
  int l, dims[2], periodic[2], in, out, nsweeps, images;
  double Delta;
  bmg_blocks B;
};

/* nsweeps red-black sweeps of a tile of one block from `in' into `out', in
   shared memory.  The window around the tile reaches into the neighbouring
   blocks, whose iterate, residual and coefficients are read where they are
   (peer memory when they live on another device): nothing is exchanged
   between the sweeps, and a cell of the window's rim, wrong from its first
   pass on, spoils one more ring per pass and never the tile.  A box side
   is folded into the weights of its cells.  A thread owns a cell of each
   colour, with its weights in registers.  The level's last launch writes
   the images.  Bound: the latency of staging a window and of eight passes.
   2 x 2 blocks of 128^2: 18.4 -> 13.0 ms per solve of 56 cycles, where a pass
   per launch took 4.2 us. */
__global__ void __launch_bounds__ (BT_THREADS, 1) k_blocks_tile (const __grid_constant__ TileParams P)
{
  __shared__ double u[2*BT_THREADS];
  const int l = P.l, n = 1 << l, ti = n < BT_I ? n : BT_I, tj = n < BT_J ? n : BT_J;
  const int b = P.B.mine[blockIdx.y], tiles = n/tj, tid = threadIdx.x;
  const bmg_blk_level * lv = P.B.lv + (long long) l*P.B.nb;
  /* the tile and its window in the domain */
  const int N[2] = {P.dims[0] << l, P.dims[1] << l};
  const int t0[2] = {((b/P.dims[1]) << l) + (int) blockIdx.x/tiles*ti,
                     ((b % P.dims[1]) << l) + (int) blockIdx.x % tiles*tj};
  int w0[2], wn[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    int hi = t0[e] + (e ? tj : ti) + BT_HALO;
    w0[e] = t0[e] - BT_HALO;
    if (!P.periodic[e]) { w0[e] = max (w0[e], 0); hi = min (hi, N[e]); }
    wn[e] = hi - w0[e];
  }
  const int nh = wn[1] >> 1, half = wn[0]*nh, row = tid/nh, h = tid - row*nh;
  const bool own = tid < half;
  double w[2][4], be[2], d[2], y[2], v[2];
  int nb[2][4], blk[2], at[2][2];
  bool plain = false;
  /* the coefficients, before the grid that this one follows is complete: it
     writes iterates and residuals only */
  if (own)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int x[2] = {row, 2*h + ((c + row) & 1)};
      int z[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        z[e] = w0[e] + x[e];
        if (P.periodic[e]) z[e] = (z[e] % N[e] + N[e]) % N[e];
        at[c][e] = z[e] & (n - 1);
      }
      blk[c] = (z[0] >> l)*P.dims[1] + (z[1] >> l);
      const bmg_blk_level & L = lv[blk[c]];
      const long long id = cidx<2> (P.g, at[c][0], at[c][1], 0);
      double dd = (-coef_of<double> (L.lambda).at (id))*(P.Delta*P.Delta);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const Coef<double> al = coef_of<double> (L.alpha[e]);
        const double w1 = al.at (id + cstride<2> (P.g, e)), wl = al.at (id);
        dd += w1 + wl;
#pragma unroll
        for (int lo = 0; lo < 2; lo++) {
          const bool box = !P.periodic[e] && z[e] == (lo ? 0 : N[e] - 1);
          const bool rim = x[e] == (lo ? 0 : wn[e] - 1);
          const double a = lo ? wl : w1;
          w[c][2*e + lo] = box && P.B.blk[blk[c]].bc.type[2*e + lo] == 1 /* BMG_DIRICHLET */ ? -a : a;
          const int m = lo ? -1 : 1;
          nb[c][2*e + lo] = rim ? c*half + tid
            : (c ^ 1)*half + (e == 0 ? (row + m)*nh + (x[1] >> 1) : row*nh + ((x[1] + m) >> 1));
        }
      }
      d[c] = dd;
      y[c] = 1./dd;
      plain = plain || divisor_unsafe (dd);
    }
  pdl_wait ();
  pdl_trigger ();
  if (own)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const bmg_blk_level & L = lv[blk[c]];
      const long long id = cidx<2> (P.g, at[c][0], at[c][1], 0);
      be[c] = (-(P.Delta*P.Delta))*L.res[id];
      v[c] = 0.;
      if (P.in == BMG_BLOCKS_DA || P.in == BMG_BLOCKS_DA2) v[c] = (P.in == BMG_BLOCKS_DA ? L.da : L.da2)[id];
      else if (P.in != BMG_BLOCKS_ZERO) {
        const bmg_blk_level & C = (lv - P.B.nb)[blk[c]];
        v[c] = bilinear<2> (P.gc, P.in == BMG_BLOCKS_COARSE_DA ? C.da : C.da2, at[c][0], at[c][1], 0);
      }
      u[c*half + tid] = v[c];
    }
  __syncthreads ();
  for (int sw = 0; sw < P.nsweeps; sw++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (own) {
        double m = be[c];
        m = m + (w[c][0]*u[nb[c][0]] + w[c][1]*u[nb[c][1]]);
        m = m + (w[c][2]*u[nb[c][2]] + w[c][3]*u[nb[c][3]]);
        v[c] = exact_quotient (m, d[c], y[c]);
        if (__any_sync (__activemask (), plain || quotient_unsafe (m))) v[c] = m/d[c];
        u[c*half + tid] = v[c];
      }
      __syncthreads ();
    }
  if (own)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int i = w0[0] + row, j = w0[1] + 2*h + ((c + row) & 1);
      if (i < t0[0] || i >= t0[0] + ti || j < t0[1] || j >= t0[1] + tj) continue;
      auto f = [=] (int t) { return P.out == BMG_BLOCKS_DA ? lv[t].da : lv[t].da2; };
      if (P.images) put<2> (P.B.blk, b, P.g, at[c][0], at[c][1], 0, v[c], true, f);
      else f (b)[cidx<2> (P.g, at[c][0], at[c][1], 0)] = v[c];
    }
}

#define NT 256

dim3 grid_of (long long threads, int m) { return dim3 ((unsigned) ((threads + NT - 1)/NT), m, 1); }

template <int DIM>
cudaError_t relax_dim (int mode, int odd, bmg_geom g, int l, bmg_blocks B, double Delta, cudaStream_t s)
{
  const long long cells = 1LL << (DIM*l);
  if (mode == BMG_SWEEP_JACOBI)
    return pdl_launch (k_blocks_relax<DIM, BMG_SWEEP_JACOBI>, grid_of (cells, B.m), dim3 (NT), 0, s, g, l, B, Delta, odd);
  if (mode == BMG_SWEEP_RED)
    return pdl_launch (k_blocks_relax<DIM, BMG_SWEEP_RED>, grid_of (cells/2, B.m), dim3 (NT), 0, s, g, l, B, Delta, 0);
  return pdl_launch (k_blocks_relax<DIM, BMG_SWEEP_BLACK>, grid_of (cells/2, B.m), dim3 (NT), 0, s, g, l, B, Delta, 0);
}

} // namespace

extern "C" {

int bmg_blocks_relax (int dim, int mode, int odd, bmg_geom g, int l, bmg_blocks B, double Delta,
                      cudaStream_t s)
{
  /* (single cells have no colours: their images would be read in the pass) */
  if (l < (mode == BMG_SWEEP_JACOBI ? 0 : 1)) return (int) cudaErrorInvalidValue;
  return status_of (dim == 1 ? relax_dim<1> (mode, odd, g, l, B, Delta, s)
                    : dim == 2 ? relax_dim<2> (mode, odd, g, l, B, Delta, s)
                    : relax_dim<3> (mode, odd, g, l, B, Delta, s));
}

int bmg_blocks_tile (bmg_geom gc, bmg_geom g, int l, bmg_blocks B, const int * dims,
                     const int * periodic, double Delta, int in, int out, int nsweeps, int images,
                     cudaStream_t s)
{
  if (l < 1 || nsweeps < 0 || nsweeps > BMG_BLOCKS_SWEEPS) return (int) cudaErrorInvalidValue;
  TileParams P;
  memset (&P, 0, sizeof P);
  P.gc = gc; P.g = g; P.l = l; P.in = in; P.out = out; P.nsweeps = nsweeps; P.images = images;
  P.Delta = Delta; P.B = B;
  for (int e = 0; e < 2; e++) { P.dims[e] = dims[e]; P.periodic[e] = periodic[e]; }
  const int n = 1 << l, ti = n < BT_I ? n : BT_I, tj = n < BT_J ? n : BT_J;
  return status_of (pdl_launch (k_blocks_tile, dim3 ((n/ti)*(n/tj), B.m, 1), dim3 (BT_THREADS), 0, s, P));
}

int bmg_blocks_prolong (int dim, int odd, bmg_geom gc, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{
  const dim3 gb = grid_of (1LL << (dim*l), B.m);
  return status_of (dim == 1 ? pdl_launch (k_blocks_prolong<1>, gb, dim3 (NT), 0, s, gc, g, l, B, odd)
                    : dim == 2 ? pdl_launch (k_blocks_prolong<2>, gb, dim3 (NT), 0, s, gc, g, l, B, odd)
                    : pdl_launch (k_blocks_prolong<3>, gb, dim3 (NT), 0, s, gc, g, l, B, odd));
}

int bmg_blocks_restrict (int dim, bmg_geom gf, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{
  const dim3 gb = grid_of (1LL << (dim*l), B.m);
  return status_of (dim == 1 ? pdl_launch (k_blocks_restrict<1>, gb, dim3 (NT), 0, s, gf, g, l, B)
                    : dim == 2 ? pdl_launch (k_blocks_restrict<2>, gb, dim3 (NT), 0, s, gf, g, l, B)
                    : pdl_launch (k_blocks_restrict<3>, gb, dim3 (NT), 0, s, gf, g, l, B));
}

int bmg_blocks_correct (int dim, int odd, bmg_geom g, int l, bmg_blocks B, cudaStream_t s)
{
  const dim3 gb = grid_of (1LL << (dim*l), B.m);
  return status_of (dim == 1 ? pdl_launch (k_blocks_correct<1>, gb, dim3 (NT), 0, s, g, l, B, odd)
                    : dim == 2 ? pdl_launch (k_blocks_correct<2>, gb, dim3 (NT), 0, s, g, l, B, odd)
                    : pdl_launch (k_blocks_correct<3>, gb, dim3 (NT), 0, s, g, l, B, odd));
}

int bmg_blocks_residual (int dim, bmg_geom g, int l, bmg_blocks B, double Delta,
                         unsigned long long * maxres, cudaStream_t s)
{
  const dim3 gb = grid_of (1LL << (dim*l), B.m);
  auto run = [&] (auto kern) { return pdl_launch (kern, gb, dim3 (NT), 0, s, g, l, B, Delta, maxres); };
  const bool p2 = delta_pow2 (Delta);
  return status_of (dim == 1 ? (p2 ? run (k_blocks_residual<1, true>) : run (k_blocks_residual<1, false>))
                    : dim == 2 ? (p2 ? run (k_blocks_residual<2, true>) : run (k_blocks_residual<2, false>))
                    : p2 ? run (k_blocks_residual<3, true>) : run (k_blocks_residual<3, false>));
}

int bmg_blocks_bottom (int dim, const bmg_geom * g, const double * Delta, int lo, int hi,
                       bmg_blocks B, const int * dims, const int * periodic, int nrelax,
                       int restrict_src, cudaStream_t s)
{
  if (lo < 1 || hi < lo || hi > BMG_MAXLEVEL) return (int) cudaErrorInvalidValue;
  BottomParams P;
  memset (&P, 0, sizeof P);
  for (int l = lo; l <= hi + (restrict_src ? 1 : 0); l++) { P.g[l] = g[l]; P.Delta[l] = Delta[l]; }
  P.B = B; P.lo = lo; P.hi = hi; P.nrelax = nrelax; P.restrict_src = restrict_src;
  const int r = dim == 1 ? staged_dim<1> (P, dims, periodic, s)
    : dim == 2 ? staged_dim<2> (P, dims, periodic, s) : staged_dim<3> (P, dims, periodic, s);
  if (r >= 0) return r;
  return status_of (dim == 1 ? pdl_launch (k_blocks_bottom<1>, dim3 (1), dim3 (1024), 0, s, P)
                    : dim == 2 ? pdl_launch (k_blocks_bottom<2>, dim3 (1), dim3 (1024), 0, s, P)
                    : pdl_launch (k_blocks_bottom<3>, dim3 (1), dim3 (1024), 0, s, P));
}

} // extern "C"
