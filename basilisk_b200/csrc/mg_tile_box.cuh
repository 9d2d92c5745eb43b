/*
 * mg_tile_box.cuh -- staging of the large 2D tiles (mg_fused.cu:
 * k_relax_tile2d_w, k_relax_tile2d_x4, k_relax_tile2d_c) along the sides of
 * the box: which cells of a thread lie on a side, and who writes which word of
 * the staged region.  Plain C++ on the host too, where a test replays it.
 *
 * A staged region is W x W cells split by colour, rows of M = W/2 per
 * colour; a thread owns 2K consecutive cells of row p, K of each colour, at
 * columns q0 = 2 m0 onwards.  The sides of the box are multiples of 2K, so
 * that these cells are inside the box or outside it together.
 *
 * Before the first pass every word has one writer between two barriers:
 * the threads outside the box zero their cells (zero_outside), and after a
 * barrier the threads inside store theirs with the ghosts that mirror them
 * (stage_cells), which lie in cells of outside threads.  In the passes
 * outside threads store nothing.
 */
#ifndef MG_TILE_BOX_CUH
#define MG_TILE_BOX_CUH

#ifdef __CUDACC__
#define BMG_HD __host__ __device__ __forceinline__
#else
#define BMG_HD inline
#endif

namespace bmgd {

template <typename T> struct alignas (16) Vec16 { T v[16/sizeof (T)]; };

/* K consecutive elements at p (16-byte aligned) */
template <typename T, int K>
BMG_HD void store_cells (T * p, const T (& v)[K])
{
  constexpr int N = 16/sizeof (T);
  static_assert (K % N == 0, "whole 16-byte words");
#pragma unroll
  for (int u = 0; u < K; u += N) {
    Vec16<T> w;
#pragma unroll
    for (int e = 0; e < N; e++) w.v[e] = v[u + e];
    *(Vec16<T> *) (p + u) = w;
  }
}

/* the sides of the box (1: below, 2: above, 4: left, 8: right) whose ghosts,
   staged in this region, mirror cells of the thread at global (gi, gj); 0
   for most threads, known for the launch */
template <int K>
BMG_HD unsigned box_sides (int gi, int gj, int p, int q0, int W, int n, int px, int py, bool ok)
{
  if (!ok) return 0;
  return (!px && gi == 0 && p > 0 ? 1u : 0u) | (!px && gi == n - 1 && p + 1 < W ? 2u : 0u) |
    (!py && gj == 0 && q0 > 0 ? 4u : 0u) | (!py && gj + 2*K == n && q0 + 2*K < W ? 8u : 0u);
}

/* the ghosts of the thread's cells of columns 2 (m0 + e) + o, values nv, in
   the array of the other colour.  Within a pass nothing inside the box reads
   a ghost but the owner of the cell that it mirrors, before it writes. */
template <int M, typename T, int K, typename B>
BMG_HD void side_ghosts (T * other, unsigned sides, int p, int m0, int o, const T (& nv)[K], const B & bc)
{
  if (!sides) return;
  T * c = other + p*M + m0;
#pragma unroll
  for (int e = 0; e < K; e++) {
    if (sides & 1u) c[e - M] = nv[e]*T(bc.fac[1]);
    if (sides & 2u) c[e + M] = nv[e]*T(bc.fac[0]);
  }
  if ((sides & 4u) && o == 0) c[-1] = nv[0]*T(bc.fac[3]);
  if ((sides & 8u) && o == 1) c[K] = nv[K - 1]*T(bc.fac[2]);
}

/* the cells of a thread outside the box: defined, though no cell inside
   reads them but for the ghosts */
template <int M, typename T, int K>
BMG_HD void zero_outside (T * even, T * odd, bool ok, int p, int m0)
{
  if (ok) return;
  const T z[K] = {};
  store_cells<T, K> (even + p*M + m0, z);
  store_cells<T, K> (odd + p*M + m0, z);
}

/* the cells of a thread inside the box, even columns in ev and odd ones in
   od, into the arrays of their colours, and their ghosts */
template <int M, typename T, int K, typename B>
BMG_HD void stage_cells (T * even, T * odd, bool ok, unsigned sides, int p, int m0, const T (& ev)[K],
                         const T (& od)[K], const B & bc)
{
  if (!ok) return;
  store_cells<T, K> (even + p*M + m0, ev);
  store_cells<T, K> (odd + p*M + m0, od);
  side_ghosts<M> (odd, sides, p, m0, 0, ev, bc);
  side_ghosts<M> (even, sides, p, m0, 1, od, bc);
}

} // namespace bmgd

#endif
