// kg_refine.cu -- Berger-Oliger transfer operators between radially nested
// levels (2:1 in r and t; the reference's mesh_refinement_lib.f90 builds a
// single uniform level, MoL/mesh_refinement_lib.f90:100-147, so refinement is
// new here).  A fine level covers [xmin, r_l] with dx_l = dx_{l-1} / 2; fine
// point ii_f sits on coarse point ii_f / 2 when ii_f is even (both grids start
// at xmin).
//   prolongation: the outermost `nbuf` fine planes take coarse values at the
//     stage time, cubic Lagrange in r, (-c(a-1) + 9 c(a) + 9 c(a+1) - c(a+2)) / 16
//     at the odd (midpoint) planes, injection at the even ones, and linear in
//     time between the coarse level's states at t and t + dt_coarse (the Pi
//     variable may live in a separate slot, as the PIRK stage arrays keep it);
//   restriction: every coarse point under the fine level's interior (all but
//     the last `keep_out` fine planes) takes the coincident fine value.
#include <cuda_runtime.h>
#include <algorithm>
#include "kg_device.cuh"
#include "kg_internal.h"
#include "kg_refine.cuh"

namespace kg {
namespace {

__global__ void prolong_kernel(Grid gf, double2* uf, double2* uf_pi, Prolong p, int nbuf) {
  pdl_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)nbuf * gf.NJ * gf.NK;
  if (t >= n) return;
  const int b = (int)(t % nbuf);
  const long long r = t / nbuf;
  const int jj = (int)(r % gf.NJ), k = (int)(r / gf.NJ);
  const int iif = gf.NI - nbuf + b;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    double2* dst = (v == 4) ? uf_pi : uf + (long long)v * gf.fs;
    dst[off3(gf, iif, jj, k)] = prolong_value(p, v, iif, jj, k);
  }
}

// the columns lo .. lo + nc - 1 of a state
__global__ void columns_kernel(Grid g, const double2* u, double2* to, int lo, int nc) {
  pdl_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nc * g.NJ * g.NK) return;
  const long long r = t / nc;
  const long long o = off3(g, lo + (int)(t % nc), (int)(r % g.NJ), (int)(r / g.NJ));
#pragma unroll
  for (int v = 0; v < 5; ++v) to[(long long)v * g.fs + o] = u[(long long)v * g.fs + o];
}

__global__ void restrict_kernel(Grid gc, double2* uc, Grid gf, const double2* uf, int nc) {
  pdl_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)nc * gc.NJ * gc.NK;
  if (t >= n) return;
  const int ic = (int)(t % nc);
  const long long r = t / nc;
  const int jj = (int)(r % gc.NJ), k = (int)(r / gc.NJ);
#pragma unroll
  for (int v = 0; v < 5; ++v)
    uc[(long long)v * gc.fs + off3(gc, ic, jj, k)] = uf[(long long)v * gf.fs + off3(gf, 2 * ic, jj, k)];
}

}  // namespace

// the stencil reaches coarse plane (NI_f - 1) / 2 + 2, which must lie inside the coarse grid
bool prolong_fits(const Grid& gf, const Grid& gc, int nbuf) {
  return nbuf >= 1 && nbuf <= gf.NI && gf.NJ == gc.NJ && gf.NK == gc.NK && (gf.NI - 1) / 2 + 2 <= gc.NI - 1 &&
         (gf.NI - nbuf) / 2 - 1 >= 0;
}

int launch_prolong(const Grid& gf, double2* uf, const Grid& gc, const double2* c_old, const double2* c_new,
                   double alpha, int nbuf, cudaStream_t st, double2* uf_pi) {
  if (!prolong_fits(gf, gc, nbuf)) return -1;
  const long long n = (long long)nbuf * gf.NJ * gf.NK;
  if (!uf_pi) uf_pi = uf + 4 * gf.fs;
  launch_pdl(prolong_kernel, (unsigned)((n + 255) / 256), 256, 0, st, gf, uf, uf_pi, Prolong{gc, c_old, c_new, alpha},
             nbuf);
  return 0;
}

// Of the coarser level's state at its step's start the prolongation reads the few
// columns about the fine level's edge, so only these are kept in the place of the
// whole state (three levels of RK4 on 512 x 33 x 65, twelve copies: 8.41 -> 8.09 ms).
void launch_keep_columns(const Grid& gc, const double2* u, double2* to, const Grid& gf, int nbuf, cudaStream_t st) {
  const int lo = std::max((gf.NI - nbuf) / 2 - 1, 0), hi = std::min((gf.NI - 1) / 2 + 2, gc.NI - 1);
  if (hi < lo) return;
  const int nc = hi - lo + 1;
  const long long n = (long long)nc * gc.NJ * gc.NK;
  launch_pdl(columns_kernel, (unsigned)((n + 255) / 256), 256, 0, st, gc, u, to, lo, nc);
}

int launch_restrict(const Grid& gc, double2* uc, const Grid& gf, const double2* uf, int keep_out, cudaStream_t st) {
  const int last_f = gf.NI - 1 - keep_out;  // last fine plane taken
  const int nc = last_f / 2 + 1;            // coarse planes 0..nc-1
  if (nc < 1 || nc > gc.NI || gf.NJ != gc.NJ || gf.NK != gc.NK) return -1;
  const long long n = (long long)nc * gc.NJ * gc.NK;
  launch_pdl(restrict_kernel, (unsigned)((n + 255) / 256), 256, 0, st, gc, uc, gf, uf, nc);
  return 0;
}

}  // namespace kg
