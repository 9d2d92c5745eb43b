/*
 * mg_tree_cycle.cu -- the correction's cycle on a quadtree in one launch of
 * one thread-block cluster, with the correction in distributed shared memory.
 *
 * The schedule interpreter (mg_tree.cu) runs a cycle as list operations on
 * global memory: between two operations the cluster barrier waits until the
 * stores have reached L2 and drops L1, so that a pass over a level costs a
 * round trip to L2 and pulls lists, coefficients and values through the
 * ports of sixteen SMs again (3 us and more per pass).  Here every cell of
 * the correction (active cells, and the halo, restricted and ghost cells
 * that a pass reads, see depend () in mg_tree_host.c) has a slot in the
 * shared memory of one CTA of the cluster; the cells of a level are dealt
 * out evenly and in order, so that most neighbours are local, and the CTA
 * that owns a cell computes it.  The coefficients, right-hand sides and
 * neighbour slots of a level's relaxation set are brought into shared memory
 * once per level (as many as fit, the others are read from global memory),
 * so a pass is local and a few remote shared-memory loads, one update per
 * thread, and a cluster barrier with no global memory in flight.
 *
 * Expressions and order are those of the interpreter's operations (relax of
 * poisson.h:303-320, bilinear and restriction of multigrid-common.h:26-32,
 * 124-140, the box conditions of common.h:957-960): the same bits.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>
#include "basilisk_mg.h"
#include "mg_device.cuh"
#include "mg_tree.h"

using namespace bmgd;

namespace {

constexpr int C = BMG_TC_RANKS, NTC = 1024;

__device__ __forceinline__ void cluster_barrier ()
{
  asm volatile ("barrier.cluster.arrive.release.aligned;\n"
                "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ uint32_t remote (uint32_t addr, uint32_t rank)
{
  uint32_t r;
  asm volatile ("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ double load_remote (uint32_t addr, double)
{
  double v;
  asm volatile ("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float load_remote (uint32_t addr, float)
{
  float v;
  asm volatile ("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ double coef (const bmg_tree_coef & c, uint32_t id) { return c.p ? c.p[id] : c.c; }
__device__ __forceinline__ float coef (const bmg_tree_coef32 & c, uint32_t id)
{
  return c.p ? c.p[id] : (float) c.c;
}

/* an item of a relaxation set: faces below and above along x and y, and
   -Delta^2 b and the diagonal */
template <typename R> struct Item { R x0, x1, y0, y1, nb, d; };
enum { I_X0 = 0, I_X1, I_Y0, I_Y1, I_NB, I_D, I_N };

template <typename R, typename CO>
struct CycleArgs {
  bmg_tc tc;
  int minlevel, maxlevel, nrelax;
  int items, cells;               /* items and stage cells held per CTA (items even) */
  const R * res;
  CO ax, ay, lam;
  double * a;
  double Delta[BMG_TREE_MAXLEVEL + 1];
  uint32_t P[BMG_TREE_MAXLEVEL + 1];
  int bctype[4];
};

template <typename R, typename CO>
__global__ void __launch_bounds__ (NTC, 1) k_tree_cycle (const __grid_constant__ CycleArgs<R, CO> A)
{
  extern __shared__ __align__ (16) unsigned char tsm[];
  R * const da = (R *) tsm;                                       /* the CTA's slots */
  /* the items one array per member (a warp's accesses are consecutive),
     then the source codes and owners of the items and of the stages' cells */
  R * const it = (R *) (tsm + ((size_t) A.tc.slots*sizeof (R) + 15)/16*16);
  uint4 * const inb = (uint4 *) (it + (size_t) I_N*A.items);
  uint32_t * const iown = (uint32_t *) (inb + A.items + A.cells);
  const uint32_t base = (uint32_t) __cvta_generic_to_shared (da);
  uint32_t me;
  asm volatile ("mov.u32 %0, %%cluster_ctarank;" : "=r"(me));
  const int tid = threadIdx.x;

  auto value = [=] (uint32_t code) -> R {
    const uint32_t r = code >> 16, o = code & 0xffffu;
    if (r == me) return da[o];
    return load_remote (remote (base + o*(uint32_t) sizeof (R), r), R (0));
  };
  auto load_item = [&] (uint32_t own, uint32_t id) {
    const int m = (int) (own >> 16);
    const R Delta = (R) A.Delta[m];
    Item<R> q;
    q.nb = - (Delta*Delta)*A.res[id];
    q.d = - coef (A.lam, id)*(Delta*Delta);
    q.x1 = coef (A.ax, id + A.P[m]); q.x0 = coef (A.ax, id);
    q.d += q.x1 + q.x0;
    q.y1 = coef (A.ay, id + 1); q.y0 = coef (A.ay, id);
    q.d += q.y1 + q.y0;
    return q;
  };

  for (int s = tid; s < A.tc.slots; s += NTC) da[s] = R (0);
  cluster_barrier ();
  for (int l = A.minlevel; l <= A.maxlevel; l++) {
    const bmg_tc_level * lv = &A.tc.lv[l];
    const uint32_t nred = lv->n[BMG_TC_RED][me], nset = nred + lv->n[BMG_TC_BLACK][me];
    const uint32_t ored = lv->off[BMG_TC_RED][me], oblk = lv->off[BMG_TC_BLACK][me];
    const int stages = lv->stages;
    uint32_t cn[BMG_TC_STAGES];
#pragma unroll
    for (int st = 0; st < BMG_TC_STAGES; st++) cn[st] = st < stages ? lv->n[BMG_TC_CELLS + st][me] : 0;
    /* the level's relaxation set: red, then black */
    for (uint32_t k = tid; k < nset && k < (uint32_t) A.items; k += NTC) {
      const uint32_t r = k < nred ? ored + k : oblk + (k - nred);
      const uint32_t own = A.tc.own[r];
      const Item<R> q = load_item (own, A.tc.id[r]);
      R * const p = it + k;
      p[I_X0*A.items] = q.x0; p[I_X1*A.items] = q.x1; p[I_Y0*A.items] = q.y0;
      p[I_Y1*A.items] = q.y1; p[I_NB*A.items] = q.nb; p[I_D*A.items] = q.d;
      inb[k] = ((const uint4 *) A.tc.src)[r];
      iown[k] = own & 0xffffu;
    }
    /* the records of its stages' cells */
    {
      uint32_t c = 0;
      for (int st = 0; st < stages; st++) {
        const uint32_t n = lv->n[BMG_TC_CELLS + st][me], o = lv->off[BMG_TC_CELLS + st][me];
        for (uint32_t k = tid; k < n && c + k < (uint32_t) A.cells; k += NTC) {
          inb[A.items + c + k] = ((const uint4 *) A.tc.src)[o + k];
          iown[A.items + c + k] = A.tc.own[o + k];
        }
        c += n;
      }
    }
    if (l == A.minlevel)
      for (uint32_t k = tid; k < nset; k += NTC)
        da[A.tc.own[k < nred ? ored + k : oblk + (k - nred)] & 0xffffu] = R (0);
    else
      for (uint32_t k = tid; k < lv->n[BMG_TC_PROLONG][me]; k += NTC) {
        const uint32_t r = lv->off[BMG_TC_PROLONG][me] + k;
        const uint4 q = ((const uint4 *) A.tc.src)[r];
        const R v = ((R) 9*value (q.x) + (R) 3*(value (q.y) + value (q.z)) + value (q.w))/(R) 16;
        da[A.tc.own[r] & 0xffffu] = v;
      }
    cluster_barrier ();
    /* the cells of each stage that the next pass reads */
    auto cells = [&] () {
      uint32_t c = 0;
#pragma unroll
      for (int st = 0; st < BMG_TC_STAGES; st++) {
        if (st >= stages) break;
        const uint32_t n = cn[st], o = lv->off[BMG_TC_CELLS + st][me];
        for (uint32_t k = tid; k < n; k += NTC) {
          const bool held = c + k < (uint32_t) A.cells;
          const uint32_t own = held ? iown[A.items + c + k] : A.tc.own[o + k], kind = own >> 16;
          const uint4 q = held ? inb[A.items + c + k] : ((const uint4 *) A.tc.src)[o + k];
          R v;
          if (kind == BMG_TC_RESTRICT) {
            R sum = 0.;
            const R v0 = value (q.x), v1 = value (q.y), v2 = value (q.z), v3 = value (q.w);
            sum += v0; sum += v1; sum += v2; sum += v3;
            v = sum/(R) (1 << 2);
          }
          else if (kind == BMG_TC_HALO) {
            const R v0 = value (q.x), v1 = value (q.y), v2 = value (q.z), v3 = value (q.w);
            v = ((R) 9*v0 + (R) 3*(v1 + v2) + v3)/(R) 16;
          }
          else {
            const double sn = value (q.x);
            const int s1 = q.y & 15, s2 = (q.y >> 4) & 15;
            double g = A.bctype[s1] == BMG_DIRICHLET ? - sn : sn;
            if ((q.y >> 8) == BMG_T_DIAGONAL)
              g = (g + (A.bctype[s2] == BMG_DIRICHLET ? - sn : sn) - sn);
            v = (R) g;
          }
          da[own & 0xffffu] = v;
        }
        c += n;
        cluster_barrier ();
      }
    };
    cells ();
    for (int sw = 0; sw < 2*A.nrelax; sw++) {
      const uint32_t k0 = sw & 1 ? nred : 0, k1 = sw & 1 ? nset : nred;
      for (uint32_t k = k0 + tid; k < k1; k += NTC) {
        Item<R> q;
        uint4 nb;
        uint32_t own;
        if (k < (uint32_t) A.items) {
          const R * const p = it + k;
          q.x0 = p[I_X0*A.items]; q.x1 = p[I_X1*A.items]; q.y0 = p[I_Y0*A.items];
          q.y1 = p[I_Y1*A.items]; q.nb = p[I_NB*A.items]; q.d = p[I_D*A.items];
          nb = inb[k];
          own = iown[k];
        }
        else {
          const uint32_t r = k < nred ? ored + k : oblk + (k - nred);
          own = A.tc.own[r];
          q = load_item (own, A.tc.id[r]);
          nb = ((const uint4 *) A.tc.src)[r];
          own &= 0xffffu;
        }
        const R xm = value (nb.x), xp = value (nb.y), ym = value (nb.z), yp = value (nb.w);
        R nn = q.nb;
        nn += q.x1*xp + q.x0*xm;
        nn += q.y1*yp + q.y0*ym;
        da[own] = nn/q.d;
      }
      cluster_barrier ();
      if (l < A.maxlevel || sw < 2*A.nrelax - 1) cells ();
    }
  }
  /* a += da: the finest level's set is the leaves */
  {
    const bmg_tc_level * lv = &A.tc.lv[A.maxlevel];
#pragma unroll
    for (int c = BMG_TC_RED; c <= BMG_TC_BLACK; c++)
      for (uint32_t k = tid; k < lv->n[c][me]; k += NTC) {
        const uint32_t r = lv->off[c][me] + k, id = A.tc.id[r];
        A.a[id] = A.a[id] + (double) da[A.tc.own[r] & 0xffffu];
      }
  }
}

template <typename R> size_t smem_of (int slots, int items, int cells)
{
  return ((size_t) slots*sizeof (R) + 15)/16*16 + (size_t) items*I_N*sizeof (R) + (size_t) (items + cells)*20;
}

/* the launch's configuration: as many of the stages' cells, then of the
   items, as fit; false when the slots do not fit or the device cannot
   schedule the cluster */
template <typename R, typename CO>
bool configure (const bmg_tc * tc, cudaLaunchConfig_t * cfg, cudaLaunchAttribute * at, int & items, int & cells)
{
  auto kern = k_tree_cycle<R, CO>;
  int dev = 0, most = 0;
  if (cudaGetDevice (&dev) != cudaSuccess ||
      cudaDeviceGetAttribute (&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError ();
    return false;
  }
  const size_t da = smem_of<R> (tc->slots, 0, 0), lim = most;
  if (da > lim || tc->slots > 65536) return false;
  cells = tc->cells;
  if (da + (size_t) cells*20 > lim) cells = (int) ((lim - da)/20);
  /* (items in fours: the arrays stay 16-byte aligned) */
  const size_t per = 4*(I_N*sizeof (R) + 20), rest = lim - da - (size_t) cells*20;
  items = (tc->items + 3)/4*4;
  if (items/4*per > rest) items = (int) (rest/per)*4;
  memset (cfg, 0, sizeof *cfg);
  cfg->gridDim = dim3 (C, 1, 1);
  cfg->blockDim = dim3 (NTC, 1, 1);
  cfg->dynamicSmemBytes = smem_of<R> (tc->slots, items, cells);
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C; at->val.clusterDim.y = 1; at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
  /* once per device */
  static int ok[64];
  if (dev < 0 || dev >= 64) return false;
  if (!ok[dev]) {
    cudaError_t e = cudaFuncSetAttribute (kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute (kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t full = *cfg;
    full.dynamicSmemBytes = most;
    int nc = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters (&nc, kern, &full);
    cudaGetLastError ();
    ok[dev] = e == cudaSuccess && nc >= 1 ? 1 : -1;
  }
  return ok[dev] > 0;
}

template <typename R, typename CO>
int launch (const bmg_tc * tc, int minlevel, int maxlevel, int nrelax, const bmg_tree_levels * T,
            const R * res, const CO * co, const bmg_tree_bc * bc, double * a, cudaStream_t st)
{
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  int items = 0, cells = 0;
  if (!configure<R, CO> (tc, &cfg, at, items, cells)) return (int) cudaErrorInvalidConfiguration;
  cfg.stream = st;
  CycleArgs<R, CO> A;
  memset (&A, 0, sizeof A);
  A.tc = *tc;
  A.minlevel = minlevel; A.maxlevel = maxlevel; A.nrelax = nrelax; A.items = items; A.cells = cells;
  A.res = res; A.ax = co[0]; A.ay = co[1]; A.lam = co[2]; A.a = a;
  for (int l = 0; l <= maxlevel; l++) { A.Delta[l] = T->Delta[l]; A.P[l] = (uint32_t) T->g[l].P; }
  for (int s = 0; s < 4; s++) A.bctype[s] = bc->type[s];
  const int e = (int) cudaLaunchKernelEx (&cfg, k_tree_cycle<R, CO>, A);
  const cudaError_t q = cudaGetLastError ();
  return e ? e : q == cudaSuccess ? 0 : (int) q;
}

} // namespace

extern "C" {

int bmg_tree_cycle_fits (const bmg_tc * tc, int mixed)
{
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  int items, cells;
  return mixed ? configure<float, bmg_tree_coef32> (tc, &cfg, at, items, cells)
    : configure<double, bmg_tree_coef> (tc, &cfg, at, items, cells);
}

int bmg_tree_launch_cycle (const bmg_tc * tc, int minlevel, int maxlevel, int nrelax,
                           const bmg_tree_levels * T, const double * res, const bmg_tree_coef * coefs,
                           const bmg_tree_bc * bc, double * a, cudaStream_t st)
{
  return launch (tc, minlevel, maxlevel, nrelax, T, res, coefs, bc, a, st);
}

int bmg_tree_launch_cycle_mixed (const bmg_tc * tc, int minlevel, int maxlevel, int nrelax,
                                 const bmg_tree_levels * T, const float * res, const bmg_tree_coef32 * coefs,
                                 const bmg_tree_bc * bc, double * a, cudaStream_t st)
{
  return launch (tc, minlevel, maxlevel, nrelax, T, res, coefs, bc, a, st);
}

} // extern "C"
