// kg_ghost.cuh -- ghost values written by the stage that forms their source.
//
// boundary() (MoL/lines_method_lib.f90:507-597) after a stage copies: the outermost
// r column from the one inside it (outflow), theta ghost rows 0..2 and NJ-3..NJ-1
// from rows 5..3 and NJ-4..NJ-6 on the plane half a turn away, plane 0 from Nz-1
// and plane Nz from 1; the excision column is 3 u1 - 3 u2 + u3.  On a state whose
// seam planes hold plane 0 = plane Nz-1 and plane Nz = plane 1 (as every fill
// leaves them), the RK stages' results on plane 0 would equal those on plane Nz-1,
// so a stage can skip plane 0 and store every result to all the points that copy
// it: no fill pass follows.  Each ghost point has one source, so it is written
// once.  (PIRK stage arrays break the seam equality at plane Nz, so the PIRK
// steppers keep the fill.)
#pragma once
#include "kg_device.cuh"

namespace kg {

// whether the thread row at (jj, k) has copies (uniform over a warp of one row)
__device__ __forceinline__ bool has_copies(const Grid& g, int jj, int k) {
  return jj <= 5 || jj >= g.NJ - 6 || k == 1 || k == g.Nzm1;
}
// the plane whose ghost rows copy plane k: k' + Nz/2 = k (mod Nz - 1), 1 <= k' < Nz,
// with plane Nz - 1 in the place of plane 0
__device__ __forceinline__ int ghost_plane(const Grid& g, int k) {
  int q = (k == g.Nzm1 ? 0 : k) - g.dis;
  if (q < 0) q += g.Nzm1;
  return q == 0 ? g.Nzm1 : q;
}
// stores val (five variables at (ii, jj, k), stored already) to its copies; next:
// also to column ii + 1
template <class T>
__device__ __forceinline__ void store_copies(const Grid& g, T* out, int ii, int jj, int k, const T (&val)[5],
                                             bool next) {
  auto put = [&](int row, int plane) {
    T* d = out + off3(g, ii, row, plane);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      d[(long long)v * g.fs] = val[v];
      if (next) d[(long long)v * g.fs + 1] = val[v];
    }
  };
  auto seam = [&](int plane) { return plane == g.Nzm1 ? 0 : plane == 1 ? g.Nz : -1; };
  const int kg = ghost_plane(g, k);
#pragma unroll 1
  for (int t = 0; t < 5; ++t) {
    // 0: the seam copy of the row itself; 1, 3: its ghost rows; 2, 4: their seam copies
    const bool north = t <= 2;
    const int row = t == 0 ? jj : north ? 5 - jj : 2 * g.NJ - 7 - jj;
    const int plane = t == 0 ? seam(k) : (t & 1) ? kg : seam(kg);
    const bool wanted = t == 0 || (north ? jj <= 5 : jj >= g.NJ - 6);
    if (wanted && plane >= 0) put(row, plane);
  }
}

}  // namespace kg
