/*
 * mg_visc.cu -- sm_100a kernels of the implicit viscous step (viscosity.h),
 * two and three dimensions, FP64, and their C launchers.
 *
 *   k_visc_pass      one colour pass (or Jacobi sweep) of relax_viscosity
 *                    (viscosity.h:25-84) over every component, from one
 *                    buffer into the other, with the boundary
 *   k_visc_bottom    the coarse end of the cycle in one CTA: restriction of
 *                    the residual, then zero / prolongation and all sweeps
 *                    of every level up to 32^2 or 8^3
 *   k_visc_restrict, k_visc_prolong, k_visc_correct
 *                    the transfer operators and u += da of all components
 *                    in one launch
 *   k_visc_residual  residual_viscosity (viscosity.h:91-160) and its maximum
 *
 * Arithmetic follows the reference's evaluation order (--fmad=false), and
 * the transfer operators that of mg_kernels.cu.
 */
#include <cuda_runtime.h>
#include <string.h>
#include "mg_launch.h"
#include "mg_device.cuh"

using namespace bmgd;

namespace {

/* components of a cell vector, and of a face coefficient */
struct VecP { double * p[3]; };
struct VecC { Coef<double> c[3]; };
struct VecB { BCH c[3]; };

/* the tangential directions of component c in foreach_dimension order
   (x -> y -> z -> x) */
template <int DIM>
__device__ __forceinline__ constexpr int vtang (int c, int m) { return DIM == 2 ? 1 - c : (c + 1 + m) % 3; }

/* the coefficients of a cell: mu on its upper and lower face of each
   direction, and dt/rho */
template <int DIM>
struct VCell {
  double mu1[DIM], mu0[DIM], s;
  __device__ __forceinline__ void load (const bmg_geom & g, const VecC & mu, const Coef<double> & rho,
                                        double dt, long long id)
  {
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      mu1[d] = mu.c[d].p ? mu.c[d].p[id + cstride<DIM> (g, d)] : mu.c[d].c;
      mu0[d] = mu.c[d].p ? mu.c[d].p[id] : mu.c[d].c;
    }
    s = dt/rho.at (id);
  }
};

/* numerator sum A and denominator sum of relax_viscosity's w.c
   (viscosity.h:36-67), lambda = 1, in the reference's evaluation order */
template <int DIM>
__device__ __forceinline__ double visc_A (const bmg_geom & g, int c, long long id, double * const * U,
                                          const VCell<DIM> & q)
{
  const long long sn = cstride<DIM> (g, c);
  const double * un = U[c];
  double A = 2.*q.mu1[c]*un[id + sn] + 2.*q.mu0[c]*un[id - sn];
#pragma unroll
  for (int m = 0; m < DIM - 1; m++) {
    const int t = vtang<DIM> (c, m);
    const long long s = cstride<DIM> (g, t);
    const double * ut = U[t];
    A = A + q.mu1[t]*(un[id + s] + (ut[id + sn] + ut[id + sn + s])/4. -
                      (ut[id - sn] + ut[id - sn + s])/4.);
    A = A - q.mu0[t]*(- un[id - s] + (ut[id + sn - s] + ut[id + sn])/4. -
                      (ut[id - sn - s] + ut[id - sn])/4.);
  }
  return A;
}

template <int DIM>
__device__ __forceinline__ double visc_den (int c, const VCell<DIM> & q)
{
  double den = 2.*q.mu1[c] + 2.*q.mu0[c];
#pragma unroll
  for (int m = 0; m < DIM - 1; m++) {
    den = den + q.mu1[vtang<DIM> (c, m)];
    den = den + q.mu0[vtang<DIM> (c, m)];
  }
  return den;
}

template <int DIM>
__device__ __forceinline__ double visc_w (const bmg_geom & g, int c, long long id, double * const * U,
                                          double R, const VCell<DIM> & q, double Delta)
{
  const double A = visc_A<DIM> (g, c, id, U, q);
  return (q.s*A + R*(Delta*Delta))/((Delta*Delta)*1. + q.s*visc_den<DIM> (c, q));
}

/* One pass of relax_viscosity over a level, from IN into OUT (the next pass
   goes back): colour 0 / 1 updates the red / black cells of every component
   from the values before the pass (the stencil reads diagonal neighbours of
   the same colour) and copies the others, JAC averages every cell with its
   update (viscosity.h:71-74); each cell writes the ghost images it has, so
   the boundary that follows a pass costs no launch.  A thread owns a pair
   of cells along the contiguous axis, one of each colour: every thread of
   a warp updates a cell.  One launch per pass where a pass used to be an
   update into a buffer, its commit and a boundary launch per component;
   on 1024^2 a pass took 26.2 + 9.1 + 2 x 5.0 us, and with the coarse levels
   in k_visc_bottom a step of 12 cycles went from 15.29 to 4.43 ms.  Bound:
   L2 (nine level arrays per pass, which fit it up to 1024^2). */
template <int DIM, bool JAC>
__global__ void k_visc_pass (bmg_geom g, int colour, VecP IN, VecP OUT, VecP R, VecC mu,
                             Coef<double> rho, double dt, double Delta, VecB bc)
{
  pdl_wait ();
  pdl_trigger ();
  int i, j, k;
  const int n = g.n;
  const int q = blockIdx.x*blockDim.x + threadIdx.x;
  if (DIM == 2) { j = 2*q; i = blockIdx.y*blockDim.y + threadIdx.y; k = 0; }
  else { k = 2*q; j = blockIdx.y*blockDim.y + threadIdx.y; i = blockIdx.z*blockDim.z + threadIdx.z; }
  if (2*q >= n || i >= n || (DIM == 3 && j >= n)) return;
  const long long id0 = cidx<DIM> (g, i, j, k);
  double v[2][DIM];                     /* the new values of the two cells */
  if (JAC) {
#pragma unroll
    for (int o = 0; o < 2; o++) {
      if (2*q + o >= n) continue;
      VCell<DIM> cf;
      cf.load (g, mu, rho, dt, id0 + o);
#pragma unroll
      for (int c = 0; c < DIM; c++)
        v[o][c] = (IN.p[c][id0 + o] +
                   2.*visc_w<DIM> (g, c, id0 + o, IN.p, R.p[c][id0 + o], cf, Delta))/3.;
    }
  }
  else {
    const int o = (colour + i + (DIM == 3 ? j : 0)) & 1;      /* the cell of this colour */
    double w[DIM], u[DIM];
    if (2*q + o < n) {
      VCell<DIM> cf;
      cf.load (g, mu, rho, dt, id0 + o);
#pragma unroll
      for (int c = 0; c < DIM; c++)
        w[c] = visc_w<DIM> (g, c, id0 + o, IN.p, R.p[c][id0 + o], cf, Delta);
    }
    if (2*q + 1 - o < n)
#pragma unroll
      for (int c = 0; c < DIM; c++) u[c] = IN.p[c][id0 + 1 - o];
#pragma unroll
    for (int c = 0; c < DIM; c++) {
      v[0][c] = o ? u[c] : w[c];
      v[1][c] = o ? w[c] : u[c];
    }
  }
#pragma unroll
  for (int c = 0; c < DIM; c++) {
    double * f = OUT.p[c];
    if (2*q + 1 < n) *(double2 *) (f + id0) = make_double2 (v[0][c], v[1][c]);
    else f[id0] = v[0][c];
    ghosts_homog<DIM, double> (f, g, i, j, k, v[0][c], bc.c[c]);
    if (2*q + 1 < n)
      ghosts_homog<DIM, double> (f, g, i, DIM == 2 ? j + 1 : j, DIM == 3 ? k + 1 : k, v[1][c], bc.c[c]);
  }
}

/* restriction_average (multigrid-common.h:26-32) of coarse cell (i, j, k)
   in foreach_child order */
template <int DIM>
__device__ __forceinline__ double visc_mean (const bmg_geom & gf, const double * f, int i, int j, int k)
{
  double sum = 0.;
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
      for (int d = 0; d < (DIM == 3 ? 2 : 1); d++)
        sum += f[cidx<DIM> (gf, 2*i + a, 2*j + b, 2*k + d)];
  return sum/(double) (1 << DIM);
}

template <int DIM>
__global__ void k_visc_restrict (bmg_geom gf, bmg_geom gc, VecP F, VecP C)
{
  pdl_wait ();
  pdl_trigger ();
  int i, j, k;
  if (!cell_of_thread<DIM> (gc.n, i, j, k)) return;
#pragma unroll
  for (int c = 0; c < DIM; c++)
    C.p[c][cidx<DIM> (gc, i, j, k)] = visc_mean<DIM> (gf, F.p[c], i, j, k);
}

/* the bilinear / trilinear prolongation (multigrid-common.h:124-140) of
   fine cell (i, j, k), in k_prolong's expression and order */
template <int DIM>
__device__ __forceinline__ double visc_bilinear (const bmg_geom & gc, const double * s, int i, int j, int k)
{
  const int pi = i >> 1, cx = (i & 1) ? 1 : -1, pj = j >> 1, cy = (j & 1) ? 1 : -1;
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
__global__ void k_visc_prolong (bmg_geom gc, bmg_geom gf, VecP C, VecP F, VecB bc)
{
  pdl_wait ();
  pdl_trigger ();
  int i, j, k;
  if (!cell_of_thread<DIM> (gf.n, i, j, k)) return;
#pragma unroll
  for (int c = 0; c < DIM; c++) {
    const double v = visc_bilinear<DIM> (gc, C.p[c], i, j, k);
    F.p[c][cidx<DIM> (gf, i, j, k)] = v;
    ghosts_homog<DIM, double> (F.p[c], gf, i, j, k, v, bc.c[c]);
  }
}

struct VecD { bmg_bcdesc c[3]; };

/* u += da with the boundary conditions of u (poisson.h:84-89) */
template <int DIM>
__global__ void k_visc_correct (bmg_geom g, VecP U, VecP DA, const __grid_constant__ VecD bc)
{
  pdl_wait ();
  pdl_trigger ();
  int i, j, k;
  if (!cell_of_thread<DIM> (g.n, i, j, k)) return;
  const long long id = cidx<DIM> (g, i, j, k);
#pragma unroll
  for (int c = 0; c < DIM; c++) {
    const double v = U.p[c][id] + DA.p[c][id];
    U.p[c][id] = v;
    ghosts_inhomog<DIM> (U.p[c], g, i, j, k, v, bc.c[c]);
  }
}

/* residual_viscosity, uniform-grid branch (viscosity.h:121-147), lambda =
   1; max |res| over the components into maxres */
template <int DIM>
__global__ void k_visc_residual (bmg_geom g, VecP U, VecP R, VecP RES, VecC mu,
                                 Coef<double> rho, double dt, double Delta,
                                 unsigned long long * maxres)
{
  pdl_wait ();
  pdl_trigger ();
  int i, j, k;
  double m = 0.;
  if (cell_of_thread<DIM> (g.n, i, j, k)) {
    const long long id = cidx<DIM> (g, i, j, k);
    VCell<DIM> q;
    q.load (g, mu, rho, dt, id);
#pragma unroll
    for (int c = 0; c < DIM; c++) {
      const long long sn = cstride<DIM> (g, c);
      const double * un = U.p[c];
      double B = 2.*q.mu1[c]*(un[id + sn] - un[id]) - 2.*q.mu0[c]*(un[id] - un[id - sn]);
#pragma unroll
      for (int e = 0; e < DIM - 1; e++) {
        const int t = vtang<DIM> (c, e);
        const long long s = cstride<DIM> (g, t);
        const double * ut = U.p[t];
        B = B + q.mu1[t]*(un[id + s] - un[id] + (ut[id + sn] + ut[id + sn + s])/4. -
                          (ut[id - sn] + ut[id - sn + s])/4.);
        B = B - q.mu0[t]*(un[id] - un[id - s] + (ut[id + sn - s] + ut[id + sn])/4. -
                          (ut[id - sn - s] + ut[id - sn])/4.);
      }
      const double r = R.p[c][id] - 1.*un[id] + q.s*B/(Delta*Delta);
      RES.p[c][id] = r;
      const double ar = fabs (r);
      if (m == m && !(ar <= m)) m = ar;       /* a NaN sticks */
    }
  }
  block_max_atomic (m, maxres);
}

/* ---------------------------------------------------------------- */
/* the coarse end of the cycle                                       */
/* ---------------------------------------------------------------- */

#define VB_THREADS 512
/* levels 0..5 in two dimensions, 0..3 in three: the cells of one colour of
   the finest of them are one per thread (two dimensions), and its correction
   fits the static shared memory twice */
template <int DIM> struct VBot { static constexpr int TOP = DIM == 2 ? 5 : 3, N = 1 << TOP; };

struct VBotParams {
  bmg_geom g[6], src;             /* levels 0..top, and level top + 1 */
  VecP res[6], src_res, da;       /* da: the result, on level top */
  VecC mu[6];
  Coef<double> rho[6];
  double Delta[6], dt;
  int top, nrelax, jacobi, restrict_src;
  VecB bc;
};

/* One CTA runs levels 0..top: the residual restricted level by level (in
   its global arrays), then per level the zero or the prolongation of the
   level below and nrelax sweeps with the correction in shared memory and
   the coefficients of a thread's cells (one of each colour) in registers.
   As one launch per pass these levels cost six to eight launches of 3 to
   5 us per sweep and level for a few hundred cells.  Bound: the latency of
   one update (its sum, a quotient through the reciprocal of the denominator,
   two barriers) per pass. */
template <int DIM>
__global__ void __launch_bounds__ (VB_THREADS, 1) k_visc_bottom (const __grid_constant__ VBotParams P)
{
  constexpr int CELLS = DIM == 2 ? (VBot<2>::N + 2)*(VBot<2>::N + 2)
                                 : (VBot<3>::N + 2)*(VBot<3>::N + 2)*(VBot<3>::N + 2);
  __shared__ double sm[2][DIM][CELLS];
  const int tid = threadIdx.x;
  pdl_wait ();
  pdl_trigger ();
  for (int m = P.restrict_src ? P.top : P.top - 1; m >= 0; m--) {
    const bmg_geom & gf = m == P.top ? P.src : P.g[m + 1];
    const VecP & F = m == P.top ? P.src_res : P.res[m + 1];
    const int total = 1 << (DIM*m);
    for (int q = tid; q < total; q += VB_THREADS) {
      const int i = q >> ((DIM - 1)*m), j = DIM == 2 ? q & ((1 << m) - 1) : (q >> m) & ((1 << m) - 1);
      const int k = DIM == 3 ? q & ((1 << m) - 1) : 0;
#pragma unroll
      for (int c = 0; c < DIM; c++)
        P.res[m].p[c][cidx<DIM> (P.g[m], i, j, k)] = visc_mean<DIM> (gf, F.p[c], i, j, k);
    }
    __syncthreads ();
  }
  bmg_geom gs, gp;                          /* shared layout of this level and the one below */
  memset (&gs, 0, sizeof gs);
  gp = gs;
  for (int m = 0; m <= P.top; m++) {
    const int n = 1 << m;
    gs.n = n; gs.P = n + 2; gs.xo = 1; gs.plane = DIM == 3 ? (n + 2)*(n + 2) : n + 2;
    double * U[DIM], * B[DIM];
#pragma unroll
    for (int c = 0; c < DIM; c++) { U[c] = sm[m & 1][c]; B[c] = sm[(m & 1) ^ 1][c]; }
    const int total = 1 << (DIM*m);
    for (int q = tid; q < total; q += VB_THREADS) {
      const int i = q >> ((DIM - 1)*m), j = DIM == 2 ? q & (n - 1) : (q >> m) & (n - 1);
      const int k = DIM == 3 ? q & (n - 1) : 0;
#pragma unroll
      for (int c = 0; c < DIM; c++) {
        const double v = m == 0 ? 0. : visc_bilinear<DIM> (gp, B[c], i, j, k);
        U[c][cidx<DIM> (gs, i, j, k)] = v;
        ghosts_homog<DIM, double> (U[c], gs, i, j, k, v, P.bc.c[c]);
      }
    }
    /* the thread's cell of each colour: coefficients, right-hand sides
       R Delta^2 and denominators */
    const double Delta = P.Delta[m];
    const int half = n > 1 ? total >> 1 : 1;
    bool own[2];
    int ci[2], cj[2], ck[2];
    VCell<DIM> cf[2];
    double rd[2][DIM], den[2][DIM], y[2][DIM];
    int goff[2][DIM], gside[2][DIM];    /* the cell's image per direction: offset (0: none), side */
    bool plain = false;                 /* a divisor outside exact_quotient's range */
#pragma unroll
    for (int o = 0; o < 2; o++) {
      own[o] = tid < (n > 1 ? half : o == 0 ? 1 : 0);
      const int lh = m > 0 ? m - 1 : 0, row = tid >> lh, h = tid & ((1 << lh) - 1);
      ci[o] = DIM == 2 ? row : row >> m;
      const int jj = DIM == 2 ? 0 : row & (n - 1), last = 2*h + ((o + ci[o] + jj) & 1);
      cj[o] = DIM == 2 ? last : jj;
      ck[o] = DIM == 2 ? 0 : last;
      if (n == 1) { ci[o] = cj[o] = ck[o] = 0; }
      if (own[o]) {
        const long long id = cidx<DIM> (P.g[m], ci[o], cj[o], ck[o]);
        cf[o].load (P.g[m], P.mu[m], P.rho[m], P.dt, id);
#pragma unroll
        for (int c = 0; c < DIM; c++) {
          rd[o][c] = P.res[m].p[c][id]*(Delta*Delta);
          den[o][c] = (Delta*Delta)*1. + cf[o].s*visc_den<DIM> (c, cf[o]);
          y[o][c] = 1./den[o][c];
          plain = plain || divisor_unsafe (den[o][c]);
        }
      }
      const int x[3] = {ci[o], cj[o], ck[o]};
#pragma unroll
      for (int e = 0; e < DIM; e++) {
        const int st = (int) cstride<DIM> (gs, e);
        const bool lo = x[e] == 0, hi = x[e] == n - 1;
        gside[o][e] = 2*e + (lo ? 1 : 0);
        goff[o][e] = !lo && !hi ? 0 : P.bc.c[0].periodic[e] ? (lo ? n : -n)*st : lo ? -st : st;
      }
    }
    /* value v of component c into cell id of colour t, and its images: all
       products of the directions' (ghosts_homog's; a single cell has two
       images per direction) */
    auto put = [&] (int t, int c, int id, double v) {
      U[c][id] = v;
      if (n == 1) { ghosts_homog<DIM, double> (U[c], gs, ci[t], cj[t], ck[t], v, P.bc.c[c]); return; }
      const int a = goff[t][0], b = goff[t][1], d = DIM == 3 ? goff[t][DIM - 1] : 0;
      if (!(a | b | d)) return;
      const BCH & h = P.bc.c[c];
      const double fa = h.periodic[0] ? 1. : h.fac[gside[t][0]], fb = h.periodic[1] ? 1. : h.fac[gside[t][1]];
      if (a) U[c][id + a] = v*fa;
      if (b) U[c][id + b] = v*fb;
      if (a && b) U[c][id + a + b] = v*fa*fb;
      if (DIM == 3 && d) {
        const double fd = h.periodic[2] ? 1. : h.fac[gside[t][DIM - 1]];
        U[c][id + d] = v*fd;
        if (a) U[c][id + a + d] = v*fa*fd;
        if (b) U[c][id + b + d] = v*fb*fd;
        if (a && b) U[c][id + a + b + d] = v*fa*fb*fd;
      }
    };
    __syncthreads ();
    for (int sw = 0; sw < P.nrelax; sw++) {
      double w[2][DIM];
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const int id = (int) cidx<DIM> (gs, ci[o], cj[o], ck[o]);
        if (own[o]) {
          double nn[DIM];
          bool unsafe = plain;
#pragma unroll
          for (int c = 0; c < DIM; c++) {
            nn[c] = cf[o].s*visc_A<DIM> (gs, c, id, U, cf[o]) + rd[o][c];
            w[o][c] = exact_quotient (nn[c], den[o][c], y[o][c]);
            unsafe = unsafe || quotient_unsafe (nn[c]);
          }
          if (__any_sync (__activemask (), unsafe))
#pragma unroll
            for (int c = 0; c < DIM; c++) w[o][c] = nn[c]/den[o][c];
        }
        /* a Jacobi sweep computes both cells before it stores either */
        if (P.jacobi && o == 0) continue;
        __syncthreads ();
#pragma unroll
        for (int t = 0; t < 2; t++) {
          if (!own[t] || (P.jacobi ? false : t != o)) continue;
          const int it = (int) cidx<DIM> (gs, ci[t], cj[t], ck[t]);
#pragma unroll
          for (int c = 0; c < DIM; c++) {
            put (t, c, it, P.jacobi ? (U[c][it] + 2.*w[t][c])/3. : w[t][c]);
          }
        }
        __syncthreads ();
      }
    }
    gp = gs;
  }
  /* da of level top, ghosts included */
  const int e = gs.n + 2, cells = DIM == 2 ? e*e : e*e*e;
  for (int q = tid; q < cells; q += VB_THREADS) {
    const int i = DIM == 2 ? q/e : q/(e*e), j = DIM == 2 ? q % e : (q/e) % e, k = DIM == 2 ? 0 : q % e;
    const long long id = cidx<DIM> (P.g[P.top], i - 1, j - 1, k - 1);
#pragma unroll
    for (int c = 0; c < DIM; c++) P.da.p[c][id] = sm[P.top & 1][c][q];
  }
}

VecP vec_of (int dim, double * const * p)
{
  VecP r;
  for (int c = 0; c < 3; c++) r.p[c] = c < dim ? p[c] : NULL;
  return r;
}

VecC coefs_of (const bmg_coef * mu)
{
  VecC r;
  for (int c = 0; c < 3; c++) r.c[c] = coef_of<double> (mu[c]);
  return r;
}

VecB bcs_of (int dim, const bmg_bcdesc * bc)
{
  VecB r;
  for (int c = 0; c < 3; c++) r.c[c] = bch_of (c < dim ? &bc[c] : NULL);
  return r;
}

int status_of (cudaError_t launched)
{
  const cudaError_t e = cudaGetLastError ();
  return launched != cudaSuccess ? (int) launched : (int) e;
}

template <int DIM>
cudaError_t pass_dim (bmg_geom g, int mode, VecP in, VecP out, VecP r, VecC mu, Coef<double> rho,
                      double dt, double Delta, VecB b, cudaStream_t s)
{
  const dim3 bb = block_shape<DIM> ();
  const int pairs = (g.n + 1)/2;
  dim3 gb ((pairs + bb.x - 1)/bb.x, (g.n + bb.y - 1)/bb.y, DIM == 3 ? (g.n + bb.z - 1)/bb.z : 1);
  if (mode == 0)
    return pdl_launch (k_visc_pass<DIM, true>, gb, bb, 0, s, g, 0, in, out, r, mu, rho, dt, Delta, b);
  return pdl_launch (k_visc_pass<DIM, false>, gb, bb, 0, s, g, mode - 1, in, out, r, mu, rho, dt, Delta, b);
}

} // namespace

extern "C" {

int bmg_launch_visc_pass (int dim, bmg_geom g, int mode, double * const * in, double * const * out,
                          double * const * r, const bmg_coef * mu, bmg_coef rho, double dt,
                          double Delta, const bmg_bcdesc * bc, cudaStream_t s)
{
  const VecP I = vec_of (dim, in), O = vec_of (dim, out), R = vec_of (dim, r);
  const VecC M = coefs_of (mu);
  const Coef<double> rh = coef_of<double> (rho);
  const VecB b = bcs_of (dim, bc);
  if (dim == 2) return status_of (pass_dim<2> (g, mode, I, O, R, M, rh, dt, Delta, b, s));
  if (dim == 3) return status_of (pass_dim<3> (g, mode, I, O, R, M, rh, dt, Delta, b, s));
  return (int) cudaErrorInvalidValue;
}

int bmg_launch_visc_residual (int dim, bmg_geom g, double * const * u, double * const * r,
                              double * const * res, const bmg_coef * mu, bmg_coef rho,
                              double dt, double Delta, unsigned long long * maxres,
                              cudaStream_t s)
{
  const VecP U = vec_of (dim, u), R = vec_of (dim, r), RES = vec_of (dim, res);
  const VecC M = coefs_of (mu);
  const Coef<double> rh = coef_of<double> (rho);
  if (dim == 2)
    return status_of (pdl_launch (k_visc_residual<2>, grid_shape<2> (g.n), block_shape<2> (), 0, s, g, U, R, RES, M, rh, dt, Delta, maxres));
  if (dim == 3)
    return status_of (pdl_launch (k_visc_residual<3>, grid_shape<3> (g.n), block_shape<3> (), 0, s, g, U, R, RES, M, rh, dt, Delta, maxres));
  return (int) cudaErrorInvalidValue;
}

int bmg_launch_visc_restrict (int dim, bmg_geom gf, bmg_geom gc, double * const * fine,
                              double * const * coarse, cudaStream_t s)
{
  const VecP F = vec_of (dim, fine), C = vec_of (dim, coarse);
  if (dim == 2)
    return status_of (pdl_launch (k_visc_restrict<2>, grid_shape<2> (gc.n), block_shape<2> (), 0, s, gf, gc, F, C));
  if (dim == 3)
    return status_of (pdl_launch (k_visc_restrict<3>, grid_shape<3> (gc.n), block_shape<3> (), 0, s, gf, gc, F, C));
  return (int) cudaErrorInvalidValue;
}

int bmg_launch_visc_prolong (int dim, bmg_geom gc, bmg_geom gf, double * const * coarse,
                             double * const * fine, const bmg_bcdesc * bc, cudaStream_t s)
{
  const VecP C = vec_of (dim, coarse), F = vec_of (dim, fine);
  const VecB b = bcs_of (dim, bc);
  if (dim == 2)
    return status_of (pdl_launch (k_visc_prolong<2>, grid_shape<2> (gf.n), block_shape<2> (), 0, s, gc, gf, C, F, b));
  if (dim == 3)
    return status_of (pdl_launch (k_visc_prolong<3>, grid_shape<3> (gf.n), block_shape<3> (), 0, s, gc, gf, C, F, b));
  return (int) cudaErrorInvalidValue;
}

int bmg_launch_visc_correct (int dim, bmg_geom g, double * const * u, double * const * da,
                             const bmg_bcdesc * bc, cudaStream_t s)
{
  const VecP U = vec_of (dim, u), D = vec_of (dim, da);
  VecD b;
  memset (&b, 0, sizeof b);
  for (int c = 0; c < dim; c++) b.c[c] = bc[c];
  if (dim == 2)
    return status_of (pdl_launch (k_visc_correct<2>, grid_shape<2> (g.n), block_shape<2> (), 0, s, g, U, D, b));
  if (dim == 3)
    return status_of (pdl_launch (k_visc_correct<3>, grid_shape<3> (g.n), block_shape<3> (), 0, s, g, U, D, b));
  return (int) cudaErrorInvalidValue;
}

int bmg_visc_bottom_top (int dim) { return dim == 2 ? VBot<2>::TOP : VBot<3>::TOP; }

int bmg_launch_visc_bottom (int dim, int top, const bmg_geom * g, double * const (* res)[3],
                            double * const * da, const bmg_coef (* mu)[3], const bmg_coef * rho,
                            const double * Delta, double dt, int nrelax, int jacobi,
                            int restrict_src, const bmg_bcdesc * bc, cudaStream_t s)
{
  if (dim < 2 || dim > 3 || top < 0 || top > bmg_visc_bottom_top (dim)) return (int) cudaErrorInvalidValue;
  VBotParams P;
  memset (&P, 0, sizeof P);
  for (int m = 0; m <= top; m++) {
    P.g[m] = g[m];
    P.res[m] = vec_of (dim, res[m]);
    P.mu[m] = coefs_of (mu[m]);
    P.rho[m] = coef_of<double> (rho[m]);
    P.Delta[m] = Delta[m];
  }
  if (restrict_src) { P.src = g[top + 1]; P.src_res = vec_of (dim, res[top + 1]); }
  P.da = vec_of (dim, da);
  P.dt = dt; P.top = top; P.nrelax = nrelax; P.jacobi = jacobi; P.restrict_src = restrict_src;
  P.bc = bcs_of (dim, bc);
  if (dim == 2) return status_of (pdl_launch (k_visc_bottom<2>, dim3 (1), dim3 (VB_THREADS), 0, s, P));
  return status_of (pdl_launch (k_visc_bottom<3>, dim3 (1), dim3 (VB_THREADS), 0, s, P));
}

} // extern "C"
