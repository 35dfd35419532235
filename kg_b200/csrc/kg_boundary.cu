// kg_boundary.cu -- ghost-zone, pole-parity and outer-boundary fills on the
// device (MoL/lines_method_lib.f90:507-597) and the Fortran <-> device layout
// conversion.
//
// The reference applies, in order: boundary_xL (third-order extrapolation into
// the excision plane), boundary_xR (outflow copy or inflow hold), boundary_yL
// and boundary_yR (theta ghost rows copied from the interior rows at phi + pi,
// no sign change), boundary_zL and boundary_zR (duplicated phi planes).
//
// The stepper path runs this as one launch over independent rows along r; each
// takes the value the whole sequence leaves there, computed from the
// pre-boundary state (see ghost_unit).
// `face` launches run one reference routine at a time (parity hook).
#include "kg_device.cuh"
#include "kg_internal.h"
#include "kg_refine.cuh"

namespace kg {

// value of u after boundary_xL / boundary_xR at (ii, jj, k)
__device__ __forceinline__ double2 xval(const Grid& g, const double2* u, const double2* up, int inflow,
                                        int ii, int jj, int k) {
  if (ii == 0)
    return cadd(csub(rmul(3.0, u[off3(g, 1, jj, k)]), rmul(3.0, u[off3(g, 2, jj, k)])), u[off3(g, 3, jj, k)]);
  if (ii == g.NI - 1) return inflow ? up[off3(g, ii, jj, k)] : u[off3(g, ii - 1, jj, k)];
  return u[off3(g, ii, jj, k)];
}

// source theta row of ghost row jj (0-based rows; rows 0..2 and NJ-3..NJ-1)
__device__ __forceinline__ int ghost_src_row(const Grid& g, int jj) {
  return (jj <= 2) ? (5 - jj) : (2 * g.NJ - 7 - jj);
}

// ---- the whole fill in one launch --------------------------------------------
// Units, each done by one thread block with its threads along r:
//   A  ghost row r of plane k, 1 <= k < Nz: the source row (js, k + pi) after the
//      x fill (6 (Nz - 1) rows);
//   C  row jj of plane 0 (from plane Nz - 1) and of plane Nz (from plane 1), ghost
//      rows through their source row (2 NJ rows);
//   B  the two x-face points of the interior rows of planes 1..Nz-1.
// No point that a unit reads is written by another one, with one exception: the
// partner of plane kp = Nz - 1 - Nz/2 is plane 0, so the ghost rows of kp take
// rows 3..5 and NJ-6..NJ-4 of plane 0 as the stage left them, and C overwrites
// those rows.  The C unit of such a row therefore reads it as well as its own
// source, and writes both copies behind a block barrier (A leaves plane kp out).
// What bounds it: on small grids the launch and the latency of a thread's loads, so
// the whole sequence is one launch and a thread requests all that it reads, both
// sources of a row of plane 0 among it, before it stores any of it; on large ones
// memory, 2 x 80 B per point of the ghost rows.  Rows longer than a block are shared
// among blocks (row_parts).  Event-timed, the faces' and rows' launch and the phi
// planes' before, and now: 64 x 17 x 33 12.8 / 10.7 us (PIRK2, x faces apart), 301 x 46
// x 90 21.0 / 12.1, 1024 x 65 x 129 43.1 / 32.0 (FP32 states 37.5 / 21.3), 2048 x 129 x
// 257 125 / 121 (PIRK2).
//
// On a refined level the outermost planes then take the coarser level's values
// (kg_refine.cuh): with WithProlong the same launch writes those instead, in A and C
// for the ghost rows and planes 0 and Nz and in B for the interior rows (384 x 33 x
// 65, four columns, us in two launches and in one: 25.9 / 17.9).  No unit reads these
// columns: the x fill of the outermost one falls away.

// excision extrapolation 3 u1 - 3 u2 + u3; FP32 stage states form it in FP64
__device__ __forceinline__ double2 excise(double2 a, double2 b, double2 c) {
  return cadd(csub(rmul(3.0, a), rmul(3.0, b)), c);
}
__device__ __forceinline__ float2 excise(float2 a, float2 b, float2 c) {
  const double2 e = excise(c2(a.x, a.y), c2(b.x, b.y), c2(c.x, c.y));
  return make_float2((float)e.x, (float)e.y);
}
__device__ __forceinline__ void hold(double2 v, double2& o) { o = v; }
__device__ __forceinline__ void hold(double2 v, float2& o) { o = make_float2((float)v.x, (float)v.y); }

template <class T>
struct Fill {
  T* u;
  const double2* up;
  int inflow;
  int cyclic;  // plane 0 was not computed and stands for plane Nz-1
};

// the values of row (js, ks) at column ii after the x fill
template <class T>
__device__ __forceinline__ void row_values(const Grid& g, const Fill<T>& F, int ii, int js, int ks, T (&v)[5]) {
  const bool outer = ii == g.NI - 1;
  const long long s = off3(g, ii == 0 ? 1 : outer ? ii - 1 : ii, js, ks);
  T b[5], c[5];
#pragma unroll
  for (int w = 0; w < 5; ++w) v[w] = F.u[w * g.fs + s];
  if (ii == 0) {
#pragma unroll
    for (int w = 0; w < 5; ++w) {
      b[w] = F.u[w * g.fs + s + 1];
      c[w] = F.u[w * g.fs + s + 2];
    }
#pragma unroll
    for (int w = 0; w < 5; ++w) v[w] = excise(v[w], b[w], c[w]);
  } else if (outer && F.inflow) {
#pragma unroll
    for (int w = 0; w < 5; ++w) hold(F.up[w * g.fs + s + 1], v[w]);
  }
}
template <class T>
__device__ __forceinline__ void store_row(const Grid& g, const Fill<T>& F, int ii, int jd, int kd, const T (&v)[5]) {
  const long long d = off3(g, ii, jd, kd);
#pragma unroll
  for (int w = 0; w < 5; ++w) F.u[w * g.fs + d] = v[w];
}

// the outermost planes of a refined level
struct NoProlong {
  static constexpr bool on = false;
  int nbuf = 0;
  __device__ void values(const Grid&, int, int, int, double2 (&)[5]) const {}
  __device__ void values(const Grid&, int, int, int, float2 (&)[5]) const {}
};
struct WithProlong {
  static constexpr bool on = true;
  Prolong p;
  int nbuf;
  __device__ void values(const Grid&, int ii, int jj, int k, double2 (&v)[5]) const {
#pragma unroll
    for (int w = 0; w < 5; ++w) v[w] = prolong_value(p, w, ii, jj, k);
  }
};

__host__ __device__ __forceinline__ int ghost_units(const Grid& g, int threads, int nbuf = 0) {
  const int faces = (2 + nbuf) * (g.NJ - 6) * (g.Nz - 1);
  return 2 * g.NJ + 6 * (g.Nz - 1) + (faces + threads - 1) / threads;
}

template <class T, class PR>
__device__ __forceinline__ void ghost_unit(const Grid& g, const Fill<T>& F, const PR& pr, int unit, int part = 0, int parts = 1) {
  const int nC = 2 * g.NJ, nA = 6 * (g.Nz - 1);
  const int end = PR::on ? g.NI - pr.nbuf : g.NI;  // columns from here on are the coarser level's
  if (unit < nC + nA) {
    int jd, kd, js, ks;
    bool both = false;  // a row of plane 0 that ghost rows of plane kp copy before it is overwritten
    if (unit < nC) {    // row jj of plane 0 or Nz
      jd = unit % g.NJ;
      const bool last = unit >= g.NJ;
      const bool ghost = jd < 3 || jd >= g.NJ - 3;
      kd = last ? g.Nz : 0;
      ks = last ? 1 : g.Nz - 1;
      js = ghost ? ghost_src_row(g, jd) : jd;
      if (ghost) ks = ktarget(g, ks);
      both = !last && !ghost && !F.cyclic && (jd <= 5 || jd >= g.NJ - 6);
    } else {  // ghost row of an inner plane
      const int q = unit - nC, r = q % 6;
      kd = 1 + q / 6;
      ks = ktarget(g, kd);
      if (ks == 0) {
        if (!F.cyclic) return;  // with plane 0's own rows
        ks = g.Nzm1;
      }
      jd = (r < 3) ? r : (g.NJ - 6 + r);
      js = ghost_src_row(g, jd);
    }
    const int kp = g.Nzm1 - g.dis;
    // the column that the outermost one copies may lie in a part of the row that is
    // overwritten before the outermost one's turn
    T edge[5];
    if (both)
#pragma unroll
      for (int w = 0; w < 5; ++w) edge[w] = F.u[w * g.fs + off3(g, g.NI - 2, jd, 0)];
    for (int i0 = part * blockDim.x; i0 < g.NI; i0 += parts * blockDim.x) {
      const int ii = i0 + threadIdx.x;
      const bool in = ii < g.NI;
      T v[5], z[5];
      if (in) {
        if (PR::on && ii >= end) pr.values(g, ii, jd, kd, v);
        else row_values(g, F, ii, js, ks, v);
        if (both) {
          if (PR::on && ii >= end) {
          } else if (ii == g.NI - 1 && !F.inflow) {
#pragma unroll
            for (int w = 0; w < 5; ++w) z[w] = edge[w];
          } else {
            row_values(g, F, ii, jd, 0, z);
          }
        }
      }
      if (both) __syncthreads();  // both rows have been read
      if (in) {
        store_row(g, F, ii, jd, kd, v);
        if (both) {
          if (jd <= 5) {
            if (PR::on && ii >= end) pr.values(g, ii, 5 - jd, kp, z);
            store_row(g, F, ii, 5 - jd, kp, z);
          }
          if (jd >= g.NJ - 6) {
            if (PR::on && ii >= end) pr.values(g, ii, 2 * g.NJ - 7 - jd, kp, z);
            store_row(g, F, ii, 2 * g.NJ - 7 - jd, kp, z);
          }
        }
      }
    }
  } else if (part == 0) {  // x-face points of the interior rows, then their columns from the coarser level
    const int f = (unit - nC - nA) * blockDim.x + threadIdx.x;
    const int nin = g.NJ - 6;
    const int sk = f / nin, jj = 3 + f % nin, sides = 2 + pr.nbuf;
    if (sk >= sides * (g.Nz - 1)) return;
    const int side = sk % sides, k = 1 + sk / sides;
    T v[5];
    if (side < 2) {
      if (PR::on && side == 1) return;
      const int ii = side ? g.NI - 1 : 0;
      row_values(g, F, ii, jj, k, v);
      store_row(g, F, ii, jj, k, v);
    } else {
      const int ii = g.NI - pr.nbuf + side - 2;
      pr.values(g, ii, jj, k, v);
      store_row(g, F, ii, jj, k, v);
    }
  }
}

// threads of a block
static int row_threads(int ni) { return ni >= 128 ? 128 : (ni + 31) / 32 * 32; }
// Blocks that share a row: one per row_threads columns, unless the outermost column
// would be alone in the last (it copies its neighbour, which must not be overwritten before).
static int row_parts(int ni) {
  const int nt = row_threads(ni);
  return ni % nt == 1 ? 1 : (ni + nt - 1) / nt;
}

// 64 registers a thread let 1024 threads run on an SM: the rows of a large grid are
// bound by the bytes in flight (1024 x 65 x 129: 31.8 us; 33.3 with 768 threads, 39.5
// with 512).  The coarser level's stencil takes 40 values at once and is the faster
// for room (384 x 33 x 65: 17.9 us with 128 registers, 20.1 with 80 or 64).  Blocks of
// 256 threads and one block a row took 15.7 us in the place of 13.8 (301 x 46 x 90).
template <class T, class PR>
__global__ void __launch_bounds__(128, PR::on ? 4 : 8) ghost_kernel(Grid g, Fill<T> F, PR pr, int unit0) {
  pdl_wait();
  ghost_unit(g, F, pr, unit0 + blockIdx.x, blockIdx.y, gridDim.y);
}

void launch_ghost_fill(const Grid& g, double2* u, const double2* up, int inflow, cudaStream_t st, bool faces_apart,
                       bool cyclic) {
  const int nt = row_threads(g.NI), parts = row_parts(g.NI), n = ghost_units(g, nt), rows = 2 * g.NJ + 6 * (g.Nz - 1);
  const Fill<double2> F = {u, up, inflow, (int)cyclic};
  auto kern = ghost_kernel<double2, NoProlong>;
  if (!faces_apart) {
    launch_pdl(kern, dim3(n, parts), nt, 0, st, g, F, NoProlong(), 0);
    return;
  }
  launch_pdl(kern, dim3(rows, parts), nt, 0, st, g, F, NoProlong(), 0);
  launch_pdl(kern, n - rows, nt, 0, st, g, F, NoProlong(), rows);
}

void launch_ghost_fill_f32(const Grid& g, float2* u, const double2* up, int inflow, cudaStream_t st) {
  const int nt = row_threads(g.NI);
  launch_pdl(ghost_kernel<float2, NoProlong>, dim3(ghost_units(g, nt), row_parts(g.NI)), nt, 0, st, g, Fill<float2>{u, up, inflow, 0},
             NoProlong(), 0);
}

void launch_ghost_prolong(const Grid& g, double2* u, const double2* up, int inflow, const Prolong& p, int nbuf,
                          cudaStream_t st) {
  const int nt = row_threads(g.NI);
  launch_pdl(ghost_kernel<double2, WithProlong>, dim3(ghost_units(g, nt, nbuf), row_parts(g.NI)), nt, 0, st,
             g, Fill<double2>{u, up, inflow, 0}, WithProlong{p, nbuf}, 0);
}

// ---- many solves at once (batched engine): one block row per solve -----------
constexpr int GB_THREADS = 128, GB_PARTS = 4;
template <class T>
__global__ void __launch_bounds__(GB_THREADS, 8) ghost_batch_kernel(const GhostDesc* __restrict__ d) {
  pdl_wait();
  const GhostDesc& D = d[blockIdx.y];
  const int parts = D.g.NI % GB_THREADS == 1 ? 1 : gridDim.z;  // see row_parts
  if ((int)blockIdx.x < ghost_units(D.g, GB_THREADS) && (int)blockIdx.z < parts)
    ghost_unit(D.g, Fill<T>{static_cast<T*>(D.u), D.up, D.inflow, 0}, NoProlong(), blockIdx.x, blockIdx.z, parts);
}

int ghost_batch_units(const Grid& g) { return ghost_units(g, GB_THREADS); }

void launch_ghost_fill_batch(const GhostDesc* d_desc, int n, int max_units, int f32, cudaStream_t st) {
  if (n <= 0) return;
  launch_pdl(f32 ? ghost_batch_kernel<float2> : ghost_batch_kernel<double2>, dim3(max_units, n, GB_PARTS), GB_THREADS, 0, st,
             d_desc);
}

// ---- one reference routine at a time ---------------------------------------
// face 0 = xL, 1 = xR, 2 = yL, 3 = yR, 4 = zL, 5 = zR
__global__ void face_kernel(Grid g, double2* u, const double2* up, int inflow, int face) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (face <= 1) {  // all (jj, k) of one x-face
    const long long n = (long long)g.NJ * g.NK;
    if (t >= n) return;
    const int jj = (int)(t % g.NJ), k = (int)(t / g.NJ);
    const int ii = face == 0 ? 0 : g.NI - 1;
    for (int v = 0; v < 5; ++v)
      u[v * g.fs + off3(g, ii, jj, k)] = xval(g, u + v * g.fs, up + v * g.fs, inflow, ii, jj, k);
  } else if (face <= 3) {  // three ghost rows of one pole, all (ii, k)
    const long long n = 3LL * g.NI * g.NK;
    if (t >= n) return;
    const int ii = (int)(t % g.NI);
    const long long rk = t / g.NI;
    const int r = (int)(rk % 3), k = (int)(rk / 3);
    const int jj = face == 2 ? r : g.NJ - 3 + r;
    const int js = ghost_src_row(g, jj), kt = ktarget(g, k);
    for (int v = 0; v < 5; ++v) u[v * g.fs + off3(g, ii, jj, k)] = u[v * g.fs + off3(g, ii, js, kt)];
  } else {  // one duplicated phi plane
    const long long n = (long long)g.NI * g.NJ;
    if (t >= n) return;
    const int ii = (int)(t % g.NI), jj = (int)(t / g.NI);
    const int kd = face == 4 ? 0 : g.Nz;
    const int ks = face == 4 ? g.Nz - 1 : 1;
    for (int v = 0; v < 5; ++v) u[v * g.fs + off3(g, ii, jj, kd)] = u[v * g.fs + off3(g, ii, jj, ks)];
  }
}

void launch_face(const Grid& g, double2* u, const double2* up, int inflow, int face, cudaStream_t st) {
  long long n = face <= 1 ? (long long)g.NJ * g.NK : face <= 3 ? 3LL * g.NI * g.NK : (long long)g.NI * g.NJ;
  face_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, u, up, inflow, face);
}

// ---- layout conversion -------------------------------------------------------
// aos: complex u(5, NI, NJ, planes k0..k1-1) (Fortran order, variable fastest);
// soa: variables 0..3 of a state, pi: its Pi variable (the PIRK stage arrays keep
// it in a slot of its own).  A block works on one (theta row, plane), so the index
// division is its own and not each thread's.  Bound by memory, 160 B a point; the
// 80-byte records pass through shared memory, so that a warp's accesses are whole
// lines on both sides (a stride of 80 B meets no bank conflict at 16 B a lane).  With
// each thread reaching for its own record, half a sector at a time, 2048 x 129 x 257
// took 2.33 ms a conversion, now 1.79 (6.4 TB/s); 1024 x 65 x 129 320 -> 248 us.
constexpr int CV = 256;
static int cv_threads(int ni) { return ni >= CV ? CV : (ni + 31) / 32 * 32; }

__global__ void __launch_bounds__(CV) aos_to_soa_kernel(Grid g, const double2* __restrict__ aos,
                                                        double2* __restrict__ soa, double2* __restrict__ pi, int k0) {
  __shared__ double2 rec[5 * CV];
  const int i0 = blockIdx.y * blockDim.x, ii = i0 + threadIdx.x;
  const int n = 5 * min((int)blockDim.x, g.NI - i0);
  const int jj = blockIdx.x % g.NJ, kk = blockIdx.x / g.NJ;
  const double2* a = aos + 5 * (((long long)kk * g.NJ + jj) * g.NI + i0);
#pragma unroll
  for (int w = 0; w < 5; ++w) {
    const int q = w * blockDim.x + threadIdx.x;
    if (q < n) rec[q] = a[q];
  }
  __syncthreads();
  if (ii >= g.NI) return;
  const long long o = off3(g, ii, jj, k0 + kk);
#pragma unroll
  for (int w = 0; w < 4; ++w) soa[w * g.fs + o] = rec[5 * threadIdx.x + w];
  pi[o] = rec[5 * threadIdx.x + 4];
}

__global__ void __launch_bounds__(CV) soa_to_aos_kernel(Grid g, const double2* __restrict__ soa,
                                                        const double2* __restrict__ pi, double2* __restrict__ aos,
                                                        int k0) {
  __shared__ double2 rec[5 * CV];
  const int i0 = blockIdx.y * blockDim.x, ii = i0 + threadIdx.x;
  const int n = 5 * min((int)blockDim.x, g.NI - i0);
  const int jj = blockIdx.x % g.NJ, kk = blockIdx.x / g.NJ;
  double2* a = aos + 5 * (((long long)kk * g.NJ + jj) * g.NI + i0);
  if (ii < g.NI) {
    const long long o = off3(g, ii, jj, k0 + kk);
    double2 v[5];
#pragma unroll
    for (int w = 0; w < 4; ++w) v[w] = soa[w * g.fs + o];
    v[4] = pi[o];
#pragma unroll
    for (int w = 0; w < 5; ++w) rec[5 * threadIdx.x + w] = v[w];
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 5; ++w) {
    const int q = w * blockDim.x + threadIdx.x;
    if (q < n) a[q] = rec[q];
  }
}

void launch_aos_to_soa(const Grid& g, const double2* aos, double2* soa, double2* pi, int k0, int k1, cudaStream_t st) {
  const int nt = cv_threads(g.NI);
  if (k1 > k0)
    aos_to_soa_kernel<<<dim3(g.NJ * (k1 - k0), (g.NI + nt - 1) / nt), nt, 0, st>>>(g, aos, soa, pi, k0);
}

void launch_soa_to_aos(const Grid& g, const double2* soa, const double2* pi, double2* aos, int k0, int k1,
                       cudaStream_t st) {
  const int nt = cv_threads(g.NI);
  if (k1 > k0)
    soa_to_aos_kernel<<<dim3(g.NJ * (k1 - k0), (g.NI + nt - 1) / nt), nt, 0, st>>>(g, soa, pi, aos, k0);
}

}  // namespace kg
