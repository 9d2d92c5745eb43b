// Replays the staging of a 64 x 64 region of the large 2D tiles on the host
// (mg_tile_box.cuh, the code of the kernels), thread by thread, for every
// position of a tile against the box: between two barriers every word has at
// most one writer, and what the first pass reads is right.  Prints the first
// fault and returns 1.
#include <cstdio>
#include <cstring>
#include <vector>
#include "mg_tile_box.cuh"

using namespace bmgd;

struct Bc { int periodic[3], fac[6]; };

static const int W = 64, M = W/2;

static int real_index (int gi, int n, int periodic)
{
  if (gi >= 0 && gi < n) return gi;
  return periodic ? (gi % n + n) % n : -1;
}

template <typename T> static T cell (int i, int j) { return (T) (1 + 1000*i + j); }

// what a thread wrote: the words of `a' that no longer hold the sentinel
template <typename T, typename F>
static void step (std::vector<T> & a, std::vector<int> & writer, int tid, F f, int & twice)
{
  std::vector<T> t (a.size (), (T) -7);
  f (t.data ());
  for (size_t w = 0; w < t.size (); w++)
    if (t[w] != (T) -7) {
      if (writer[w] >= 0 && writer[w] != tid && twice < 0) twice = (int) w;
      writer[w] = tid;
      a[w] = t[w];
    }
}

template <typename T, int K>
static int region (int n, int TS, int by, int bx, const Bc & bc)
{
  const int H = (W - TS)/2, i0 = by*TS - H, j0 = bx*TS - H, base = (i0 + j0) & 1;
  const int px = bc.periodic[0], py = bc.periodic[1], cols = W/(2*K);
  // (a row of guard words on either side: the neighbours' columns at its ends)
  std::vector<T> a (2*W*M + 2*M, (T) -7);
  std::vector<int> zeroed (a.size (), -1), staged (a.size (), -1);
  int twice = -1;
  for (int phase = 0; phase < 2; phase++)          // a barrier between the two
    for (int tid = 0; tid < W*cols; tid++) {
      const int p = tid/cols, q0 = 2*K*(tid % cols), m0 = q0/2, cq = (base + p) & 1;
      const int ri = real_index (i0 + p, n, px), rj = real_index (j0 + q0, n, py);
      const bool ok = ri >= 0 && rj >= 0;
      const unsigned sides = box_sides<K> (i0 + p, j0 + q0, p, q0, W, n, px, py, ok);
      T ev[K], od[K];
      for (int e = 0; e < K; e++) {
        ev[e] = ok ? cell<T> (ri, rj + 2*e) : T (0);
        od[e] = ok ? cell<T> (ri, rj + 2*e + 1) : T (0);
      }
      step (a, phase ? staged : zeroed, tid, [&] (T * t) {
        T * even = t + M + cq*W*M, * odd = t + M + (cq ^ 1)*W*M;
        if (phase == 0) zero_outside<M, T, K> (even, odd, ok, p, m0);
        else stage_cells<M> (even, odd, ok, sides, p, m0, ev, od, bc);
      }, twice);
    }
  if (twice >= 0) {
    printf ("n %d tile %d (%d, %d) periodic %d %d: word %d has two writers between barriers\n", n, TS, by,
            bx, px, py, twice);
    return 1;
  }
  for (int p = 0; p < W; p++)
    for (int q = 0; q < W; q++) {
      const int gi = i0 + p, gj = j0 + q, w = M + ((base + p + q) & 1)*W*M + p*M + q/2;
      int ri = real_index (gi, n, px), rj = real_index (gj, n, py), f = 1;
      T want = 0;
      if (ri < 0 && rj >= 0 && (gi == -1 || gi == n)) {        // the ghosts of the box
        f = bc.fac[gi < 0 ? 1 : 0];
        ri = gi < 0 ? 0 : n - 1;
        // (its mirror is staged, or the ghost is the region's rim)
        if (p + (gi < 0 ? 1 : -1) < 0 || p + (gi < 0 ? 1 : -1) >= W) continue;
      }
      else if (rj < 0 && ri >= 0 && (gj == -1 || gj == n)) {
        f = bc.fac[gj < 0 ? 3 : 2];
        rj = gj < 0 ? 0 : n - 1;
        if (q + (gj < 0 ? 1 : -1) < 0 || q + (gj < 0 ? 1 : -1) >= W) continue;
      }
      if (ri >= 0 && rj >= 0) want = cell<T> (ri, rj)*(T) f;
      if (a[w] != want) {
        printf ("n %d tile %d (%d, %d) periodic %d %d: cell (%d, %d) holds %g, not %g\n", n, TS, by, bx, px,
                py, gi, gj, (double) a[w], (double) want);
        return 1;
      }
    }
  return 0;
}

template <typename T, int K>
static int all (int n, int TS)
{
  const int tiles = (n + TS - 1)/TS;
  for (int per = 0; per < 4; per++) {
    const Bc bc = {{per & 1, per >> 1, 0}, {-1, 1, 1, -1, 1, 1}};
    for (int by = 0; by < tiles; by++)
      for (int bx = 0; bx < tiles; bx++) {
        // the tiles near a side, and one inside
        const bool ey = by < 2 || by >= tiles - 2, ex = bx < 2 || bx >= tiles - 2;
        if ((ey || by == 3) && (ex || bx == 3) && region<T, K> (n, TS, by, bx, bc)) return 1;
      }
  }
  return 0;
}

int main ()
{
  for (int n = 512; n <= 1024; n *= 2)       // (the remainders of n by a tile)
    if (all<float, 4> (n, 48) || all<float, 4> (n, 32) || all<double, 2> (n, 48) || all<double, 4> (n, 48))
      return 1;
  return 0;
}
