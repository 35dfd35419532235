// kg_refine.cuh -- value of a refined level's outermost planes from the coarser
// level (see kg_refine.cu), shared by the transfer kernel and the ghost fill.
#pragma once
#include "kg_device.cuh"

namespace kg {

struct Prolong {
  Grid gc;                 // the coarser level
  const double2* c_old;    // its state at its step's start and end
  const double2* c_new;
  double alpha;            // time in between, 0..1
};

__device__ __forceinline__ double2 prolong_r(const Grid& gc, const double2* c, int iif, int jj, int k) {
  if ((iif & 1) == 0) return c[off3(gc, iif >> 1, jj, k)];
  const int a = iif >> 1;
  const double2 cm = c[off3(gc, a - 1, jj, k)], c0 = c[off3(gc, a, jj, k)], c1 = c[off3(gc, a + 1, jj, k)],
                c2v = c[off3(gc, a + 2, jj, k)];
  return rmul(1.0 / 16.0, csub(cadd(cadd(cneg(cm), rmul(9.0, c0)), rmul(9.0, c1)), c2v));
}
// variable v at fine column iif, cubic in r and linear in time
__device__ __forceinline__ double2 prolong_value(const Prolong& p, int v, int iif, int jj, int k) {
  const double2 po = prolong_r(p.gc, p.c_old + (long long)v * p.gc.fs, iif, jj, k);
  const double2 pn = prolong_r(p.gc, p.c_new + (long long)v * p.gc.fs, iif, jj, k);
  return cadd(rmul(1.0 - p.alpha, po), rmul(p.alpha, pn));
}

}  // namespace kg
