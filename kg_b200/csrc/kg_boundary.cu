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
// those rows.  The C unit of such a row therefore writes kp's ghost rows first
// and the row itself behind a block barrier (A leaves plane kp out).
// What bounds it: on small grids the launch and the latency of one load-store
// chain per thread, so one launch replaces the former two (ghost rows and faces,
// then the phi planes); on large ones memory, 2 x 80 B per point of the ghost rows.
// Event-timed, two launches before and one after: 301 x 46 x 90 21.5 -> 17.1 us,
// 1024 x 65 x 129 43.1 -> 33.9 us (FP32 states 37.4 -> 22.1 us).  With the x faces
// apart (PIRK2) 64 x 17 x 33 13.0 -> 12.1 us, 2048 x 129 x 257 123.8 -> 119.9 us.
template <class T>
__device__ __forceinline__ T xval_t(const Grid& g, const T* u, const double2* up, int inflow, int ii, int jj, int k);
template <>
__device__ __forceinline__ double2 xval_t<double2>(const Grid& g, const double2* u, const double2* up, int inflow,
                                                   int ii, int jj, int k) {
  return xval(g, u, up, inflow, ii, jj, k);
}
// FP32 stage states: the excision extrapolation is formed in FP64, the inflow
// hold reads u^n (FP64)
template <>
__device__ __forceinline__ float2 xval_t<float2>(const Grid& g, const float2* u, const double2* up, int inflow, int ii,
                                                 int jj, int k) {
  if (ii == 0) {
    const float2 a = u[off3(g, 1, jj, k)], b = u[off3(g, 2, jj, k)], c = u[off3(g, 3, jj, k)];
    const double rx = (3.0 * (double)a.x - 3.0 * (double)b.x) + (double)c.x;
    const double ry = (3.0 * (double)a.y - 3.0 * (double)b.y) + (double)c.y;
    return make_float2((float)rx, (float)ry);
  }
  if (ii == g.NI - 1) {
    if (inflow) {
      const double2 v = up[off3(g, ii, jj, k)];
      return make_float2((float)v.x, (float)v.y);
    }
    return u[off3(g, ii - 1, jj, k)];
  }
  return u[off3(g, ii, jj, k)];
}

// row (jd, kd) <- row (js, ks) after the x fill, all five variables
template <class T>
__device__ __forceinline__ void ghost_row(const Grid& g, T* u, const double2* up, int inflow, int jd, int kd, int js,
                                          int ks) {
  const long long d = off3(g, 0, jd, kd), s = off3(g, 0, js, ks);
  for (int ii = threadIdx.x; ii < g.NI; ii += blockDim.x) {
    T v[5];
    if (ii == 0 || ii == g.NI - 1) {
#pragma unroll
      for (int w = 0; w < 5; ++w) v[w] = xval_t<T>(g, u + w * g.fs, up + w * g.fs, inflow, ii, js, ks);
    } else {
#pragma unroll
      for (int w = 0; w < 5; ++w) v[w] = u[w * g.fs + s + ii];
    }
#pragma unroll
    for (int w = 0; w < 5; ++w) u[w * g.fs + d + ii] = v[w];
  }
}

__host__ __device__ __forceinline__ int ghost_units(const Grid& g, int threads) {
  const int faces = 2 * (g.NJ - 6) * (g.Nz - 1);
  return 2 * g.NJ + 6 * (g.Nz - 1) + (faces + threads - 1) / threads;
}

template <class T>
__device__ __forceinline__ void ghost_unit(const Grid& g, T* u, const double2* up, int inflow, int unit,
                                           int cyclic = 0) {
  const int nC = 2 * g.NJ, nA = 6 * (g.Nz - 1);
  if (unit < nC) {  // row jj of plane 0 or Nz
    const int jj = unit % g.NJ;
    const bool last = unit >= g.NJ;
    const int ks = last ? 1 : g.Nz - 1;
    const bool ghost = jj < 3 || jj >= g.NJ - 3;
    if (!last && !ghost && !cyclic) {
      const int kp = g.Nzm1 - g.dis;
      const bool north = jj <= 5, south = jj >= g.NJ - 6;
      if (north) ghost_row(g, u, up, inflow, 5 - jj, kp, jj, 0);
      if (south) ghost_row(g, u, up, inflow, 2 * g.NJ - 7 - jj, kp, jj, 0);
      if (north || south) __syncthreads();
    }
    ghost_row(g, u, up, inflow, jj, last ? g.Nz : 0, ghost ? ghost_src_row(g, jj) : jj, ghost ? ktarget(g, ks) : ks);
  } else if (unit < nC + nA) {  // ghost row of an inner plane
    const int q = unit - nC;
    const int r = q % 6, k = 1 + q / 6;
    int kt = ktarget(g, k);
    if (kt == 0) {
      if (!cyclic) return;  // with plane 0's own rows
      kt = g.Nzm1;          // plane 0 was not computed: it equals plane Nz - 1
    }
    const int jj = (r < 3) ? r : (g.NJ - 6 + r);
    ghost_row(g, u, up, inflow, jj, k, ghost_src_row(g, jj), kt);
  } else {  // x-face points
    const int f = (unit - nC - nA) * blockDim.x + threadIdx.x;
    const int nin = g.NJ - 6;
    if (f >= 2 * nin * (g.Nz - 1)) return;
    const int jj = 3 + f % nin, sk = f / nin;
    const int k = 1 + (sk >> 1), ii = (sk & 1) ? g.NI - 1 : 0;
#pragma unroll
    for (int w = 0; w < 5; ++w)
      u[w * g.fs + off3(g, ii, jj, k)] = xval_t<T>(g, u + w * g.fs, up + w * g.fs, inflow, ii, jj, k);
  }
}

// threads of a block: a row of a small grid in one pass, 256 for longer rows
static int row_threads(int ni) { return ni >= 256 ? 256 : (ni + 31) / 32 * 32; }

template <class T>
__global__ void ghost_kernel(Grid g, T* u, const double2* up, int inflow, int unit0, int cyclic) {
  pdl_wait();
  ghost_unit(g, u, up, inflow, unit0 + blockIdx.x, cyclic);
}

void launch_ghost_fill(const Grid& g, double2* u, const double2* up, int inflow, cudaStream_t st, bool faces_apart,
                       bool cyclic) {
  const int nt = row_threads(g.NI), n = ghost_units(g, nt), rows = 2 * g.NJ + 6 * (g.Nz - 1);
  if (!faces_apart) {
    launch_pdl(ghost_kernel<double2>, n, nt, 0, st, g, u, up, inflow, 0, (int)cyclic);
    return;
  }
  launch_pdl(ghost_kernel<double2>, rows, nt, 0, st, g, u, up, inflow, 0, (int)cyclic);
  launch_pdl(ghost_kernel<double2>, n - rows, nt, 0, st, g, u, up, inflow, rows, (int)cyclic);
}

void launch_ghost_fill_f32(const Grid& g, float2* u, const double2* up, int inflow, cudaStream_t st) {
  const int nt = row_threads(g.NI);
  launch_pdl(ghost_kernel<float2>, ghost_units(g, nt), nt, 0, st, g, u, up, inflow, 0, 0);
}

// ---- many solves at once (batched engine): one block row per solve -----------
constexpr int GB_THREADS = 128;
template <class T>
__global__ void ghost_batch_kernel(const GhostDesc* __restrict__ d) {
  pdl_wait();
  const GhostDesc& D = d[blockIdx.y];
  if ((int)blockIdx.x < ghost_units(D.g, GB_THREADS))
    ghost_unit(D.g, static_cast<T*>(D.u), D.up, D.inflow, blockIdx.x);
}

int ghost_batch_units(const Grid& g) { return ghost_units(g, GB_THREADS); }

void launch_ghost_fill_batch(const GhostDesc* d_desc, int n, int max_units, int f32, cudaStream_t st) {
  if (n <= 0) return;
  launch_pdl(f32 ? ghost_batch_kernel<float2> : ghost_batch_kernel<double2>, dim3(max_units, n), GB_THREADS, 0, st,
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
// division is its own and not each thread's; consecutive threads touch
// consecutive 80-byte records.
__global__ void aos_to_soa_kernel(Grid g, const double2* __restrict__ aos, double2* __restrict__ soa,
                                  double2* __restrict__ pi, int k0) {
  const int ii = blockIdx.y * blockDim.x + threadIdx.x;
  if (ii >= g.NI) return;
  const int jj = blockIdx.x % g.NJ, kk = blockIdx.x / g.NJ;
  const double2* a = aos + 5 * (((long long)kk * g.NJ + jj) * g.NI + ii);
  const long long o = off3(g, ii, jj, k0 + kk);
  double2 v[5];
#pragma unroll
  for (int w = 0; w < 5; ++w) v[w] = a[w];
#pragma unroll
  for (int w = 0; w < 4; ++w) soa[w * g.fs + o] = v[w];
  pi[o] = v[4];
}

__global__ void soa_to_aos_kernel(Grid g, const double2* __restrict__ soa, const double2* __restrict__ pi,
                                  double2* __restrict__ aos, int k0) {
  const int ii = blockIdx.y * blockDim.x + threadIdx.x;
  if (ii >= g.NI) return;
  const int jj = blockIdx.x % g.NJ, kk = blockIdx.x / g.NJ;
  double2* a = aos + 5 * (((long long)kk * g.NJ + jj) * g.NI + ii);
  const long long o = off3(g, ii, jj, k0 + kk);
  double2 v[5];
#pragma unroll
  for (int w = 0; w < 4; ++w) v[w] = soa[w * g.fs + o];
  v[4] = pi[o];
#pragma unroll
  for (int w = 0; w < 5; ++w) a[w] = v[w];
}

void launch_aos_to_soa(const Grid& g, const double2* aos, double2* soa, double2* pi, int k0, int k1, cudaStream_t st) {
  const int nt = row_threads(g.NI);
  if (k1 > k0)
    aos_to_soa_kernel<<<dim3(g.NJ * (k1 - k0), (g.NI + nt - 1) / nt), nt, 0, st>>>(g, aos, soa, pi, k0);
}

void launch_soa_to_aos(const Grid& g, const double2* soa, const double2* pi, double2* aos, int k0, int k1,
                       cudaStream_t st) {
  const int nt = row_threads(g.NI);
  if (k1 > k0)
    soa_to_aos_kernel<<<dim3(g.NJ * (k1 - k0), (g.NI + nt - 1) / nt), nt, 0, st>>>(g, soa, pi, aos, k0);
}

}  // namespace kg
