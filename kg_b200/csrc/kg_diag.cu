// kg_diag.cu -- diagnostics of MoL/diagnostic_lib.f90 on the device:
// energy density, the trapezium-weighted mass integral, the ADM currents and
// detector fluxes, and the Y_lm projection at the detector radii.
//
// All reductions are deterministic: each block reduces its slice with warp
// shuffles (FP64) into one partial, and a single block adds the partials in
// a fixed order.  In the mass integral that is the block that finishes last,
// elected by an atomic counter: which block adds depends on the scheduling, the
// order of the additions and so the result do not.
#include "kg_device.cuh"
#include "kg_internal.h"
#include "kg_diag.h"

namespace kg {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double2 warp_sum2(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  return v;
}
// block-wide sum (blockDim.x multiple of 32, <= 1024); result valid in thread 0
__device__ double block_sum(double v) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
  if (w == 0) v = warp_sum(v);
  __syncthreads();
  return v;
}
__device__ double2 block_sum2(double2 v) {
  __shared__ double2 sh2[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum2(v);
  if (lane == 0) sh2[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  v = (threadIdx.x < nw) ? sh2[threadIdx.x] : make_double2(0.0, 0.0);
  if (w == 0) v = warp_sum2(v);
  __syncthreads();
  return v;
}

// density (diagnostic_lib.f90:277-289); the complex term 2 g^rphi |psi1| psi3
// makes the sum complex and rho keeps its real part.
__global__ void density_kernel(Grid g, Metric m, const double2* u, double mass2, double* rho) {
  pdl_wait();
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  const int jj = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (ii >= g.NI || jj >= g.NJ || k >= g.NK) return;
  const long long p = off3(g, ii, jj, k);
  const int q = off2(g, ii, jj);
  const double2 u1 = u[p], u2 = u[g.fs + p], u3 = u[2 * g.fs + p], u4 = u[3 * g.fs + p], u5 = u[4 * g.fs + p];
  const double a5 = hypot(u5.x, u5.y), a2 = hypot(u2.x, u2.y), a3 = hypot(u3.x, u3.y);
  const double a4 = hypot(u4.x, u4.y), a1 = hypot(u1.x, u1.y);
  const double t1 = m.grr[q] * (a2 * a2);
  const double t2re = (2.0 * m.grp[q] * a2) * u4.x;
  const double t3 = m.gtt[q] * (a3 * a3);
  const double t4 = m.gpp[q] * (a4 * a4);
  const double t5 = mass2 * a1;
  double re = a5 + t1;
  re = re + t2re;
  re = re + t3;
  re = re + t4;
  re = re + t5;
  rho[p] = 0.5 * re;
}

void launch_density(const Grid& g, const Metric& m, const double2* u, double mass2, double* rho, cudaStream_t st) {
  dim3 b(64, 4, 1), gr((g.NI + 63) / 64, (g.NJ + 3) / 4, g.NK);
  launch_pdl(density_kernel, gr, b, 0, st, g, m, u, mass2, rho);
}

// trapezium over i in [0,Nx] (ii in [2, NI-3]), j in [0,Ny], k in [0,Nz] of
// rho*sqrtg, weights 1/2 on the first and last index of each direction
static const int MASS_THREADS = 256;
int mass_blocks(const Grid& g) { return 148 * 4; }  // one wave at 4 CTAs (64 registers) per SM

// Each warp takes whole (theta, phi) rows in turn and its lanes stride along r
// with eight independent loads of rho (and of sqrt(gamma)) in flight, so the
// loads are coalesced and no per-point index division is needed; the block
// count follows from the grid, so the partial sums (and the result) do not depend
// on the device.
// One launch: the CTA that finishes last (a counter behind a fence, cleared for
// the next call) adds the partials in a fixed order.  A grid with fewer than 8 rows
// for each CTA of a full wave launches fewer.
struct MassSum {
  double value;
  unsigned int left;
};
__global__ void mass_kernel(Grid g, const double* sqrtg, const double* rho, double* partials, MassSum* sum,
                            double scale, double* host) {
  pdl_wait();
  const int ni = g.NI - 4, nj = g.NJ - 4, nk = g.NK;
  const int rows = nj * nk;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double acc = 0.0;
  for (int row = blockIdx.x * nw + (threadIdx.x >> 5); row < rows; row += gridDim.x * nw) {
    const int b = row % nj, k = row / nj;
    const int jj = b + 2;
    double wjk = 1.0;
    if (b == 0 || b == nj - 1) wjk *= 0.5;
    if (k == 0 || k == nk - 1) wjk *= 0.5;
    const double* rr = rho + off3(g, 2, jj, k);
    const double* sr = sqrtg + off2(g, 2, jj);
    for (int a0 = lane; a0 < ni; a0 += 256) {
      double rv[8], sv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int a = a0 + 32 * u;
        rv[u] = a < ni ? rr[a] : 0.0;
        sv[u] = a < ni ? __ldg(sr + a) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int a = a0 + 32 * u;
        const double w = (a == 0 || a == ni - 1) ? 0.5 * wjk : wjk;
        acc += w * (rv[u] * sv[u]);
      }
    }
  }
  acc = block_sum(acc);
  __shared__ int last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = acc;
    __threadfence();
    last = atomicAdd(&sum->left, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // 1024 strided sums and their tree, by 256 threads of four sums each
  double t4[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    t4[q] = 0.0;
    for (int i = threadIdx.x + MASS_THREADS * q; i < (int)gridDim.x; i += 4 * MASS_THREADS) t4[q] += __ldcg(partials + i);
  }
  // warp w of 32 held threads 32 w .. 32 w + 31: here warps 0..7 hold eight of them per q
  __shared__ double ws[32];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double v = warp_sum(t4[q]);
    if (lane == 0) ws[(threadIdx.x >> 5) + 8 * q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double v = warp_sum(ws[threadIdx.x]);
    if (threadIdx.x == 0) {
      sum->value = v * scale;
      if (host) *host = v * scale;
      sum->left = 0u;
    }
  }
}

void launch_mass(const Grid& g, const Metric& m, const double* rho, double dxdydz, double* partials, double* out,
                 double* host, cudaStream_t st) {
  const long long rows = (long long)(g.NJ - 4) * g.NK;
  const int nw = MASS_THREADS / 32;
  const int nb = (int)(rows < (long long)nw * mass_blocks(g) ? (rows + nw - 1) / nw : mass_blocks(g));
  launch_pdl(mass_kernel, nb, MASS_THREADS, 0, st, g, m.sqrtg, rho, partials, reinterpret_cast<MassSum*>(out), dxdydz,
             host);
}

// ---- detector shells ---------------------------------------------------------
// Vertex values of one field on the detector shells by the reference's
// trilinear interpolation (tools/FFT_sph.f90:525-651).  The index search and
// the weights depend only on the vertex index in each direction; they are
// computed once on the host with the reference's arithmetic and passed in.
//   src: 0 = phi, 1..3 = j_i * sqrtg (currents_ADM, diagnostic_lib.f90:219-229)
// One thread forms every field asked for (bit 0: phi, bits 1..3: the currents)
// at its vertex: the eight corners' values are loaded once, as independent loads.
// The kernel is bound by that one latency on the grids that are sampled every few
// steps: four fields on 64 x 17 x 33, five detectors, event-timed us in a launch per
// field and in one: 31 / 8.7.
template <int MASK>
__global__ void shell_interp_kernel(Grid g, Metric m, const double2* u, ShellInterp si, int Ny, int Nz,
                                    double2* out) {
  pdl_wait();
  constexpr int NF = MASK == 1 ? 1 : (MASK & 1) ? 4 : 3, F0 = (MASK & 1) ? 0 : 1;  // fields F0 .. F0 + NF - 1
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int d = blockIdx.y;
  if (t >= Ny * Nz || !si.active[d]) return;
  const int jv = t % Ny, kv = t / Ny;
  const int ir = si.i_r[d], ith = si.i_th[jv], iph = si.i_ph[kv];
  double2* o = out + (long long)d * 4 * Ny * Nz + t;
  // the fields at one stored point (currents_ADM, diagnostic_lib.f90:219-229)
  auto src = [&](int ii, int jj, int k, double2 (&f)[NF]) {
    const long long p = off3(g, ii, jj, k);
    if (MASK & 1) f[0] = u[p];
    if (MASK & 14) {
      const int q = off2(g, ii, jj);
      const double2 u2 = u[g.fs + p], u3 = u[2 * g.fs + p], u4 = u[3 * g.fs + p], u5 = u[4 * g.fs + p];
      const double2 n5 = cneg(u5);
      const double sg = m.sqrtg[q], grp = m.grp[q];
      const double2 a[3] = {cadd(rmul(m.grr[q], u2), rmul(grp, u4)), rmul(m.gtt[q], u3),
                            cadd(rmul(grp, u2), rmul(m.gpp[q], u4))};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double2 j = c2(n5.x * a[c].x - n5.y * a[c].y, n5.x * a[c].y + n5.y * a[c].x);
        f[NF - 3 + c] = c2(j.x * sg, j.y * sg);
      }
    }
  };
  const int fl = si.th_flag[jv];
  if (fl) {
    double2 f[NF];
    src(ir, fl == 1 ? 0 : g.NJ - 1, iph, f);
#pragma unroll
    for (int v = 0; v < NF; ++v) o[(long long)(F0 + v) * Ny * Nz] = f[v];
    return;
  }
  const double wr = si.w_r[d], wt = si.w_th[jv], wp = si.w_ph[kv];
  double2 c[8][NF];  // corners, bits: r, theta, phi
#pragma unroll
  for (int q = 0; q < 8; ++q) src(ir + (q >> 2), ith + ((q >> 1) & 1), iph + (q & 1), c[q]);
#pragma unroll
  for (int v = 0; v < NF; ++v) {
    const double2 f00 = cadd(rmul(1.0 - wp, c[0][v]), rmul(wp, c[1][v]));
    const double2 f01 = cadd(rmul(1.0 - wp, c[2][v]), rmul(wp, c[3][v]));
    const double2 f10 = cadd(rmul(1.0 - wp, c[4][v]), rmul(wp, c[5][v]));
    const double2 f11 = cadd(rmul(1.0 - wp, c[6][v]), rmul(wp, c[7][v]));
    const double2 f0 = cadd(rmul(1.0 - wt, f00), rmul(wt, f01));
    const double2 f1 = cadd(rmul(1.0 - wt, f10), rmul(wt, f11));
    o[(long long)(F0 + v) * Ny * Nz] = cadd(rmul(1.0 - wr, f0), rmul(wr, f1));
  }
}

void launch_shell_interp(const Grid& g, const Metric& m, const double2* u, const ShellInterp& si, int n_det, int Ny,
                         int Nz, int which_mask, double2* out, cudaStream_t st) {
  const int nt = 64;  // a vertex sphere of a small grid still spreads over the SMs
  dim3 gr((Ny * Nz + nt - 1) / nt, n_det);
  launch_pdl(which_mask == 1 ? shell_interp_kernel<1> : which_mask == 14 ? shell_interp_kernel<14> : shell_interp_kernel<15>,
             gr, nt, 0, st, g, m, u, si, Ny, Nz, out);
}

// trapezium_2D_complex selector weight (tools/integral.f90:330-362)
__device__ __forceinline__ double trap_w(int jv, int kv, int Ny, int Nz) {
  const int sel = ((jv == 0 || jv == Ny - 1) ? 1 : 0) + 2 * ((kv == 0 || kv == Nz - 1) ? 1 : 0);
  return sel == 0 ? 1.0 : (sel == 3 ? 0.25 : 0.5);
}

// momentum(c, d) = Re trapezium_2D(shell of j_c sqrtg): one block per (c, d)
__device__ __forceinline__ void flux_block(const double2* shells, int c, int d, int Ny, int Nz, double dydz,
                                           double* out) {
  const double2* f = shells + ((long long)d * 4 + 1 + c) * Ny * Nz;
  double2 acc = c2(0.0, 0.0);
  for (int t = threadIdx.x; t < Ny * Nz; t += blockDim.x) {
    const int jv = t % Ny, kv = t / Ny;
    acc = cadd(acc, rmul(trap_w(jv, kv, Ny, Nz), f[t]));
  }
  acc = block_sum2(acc);
  if (threadIdx.x == 0) out[c + 3 * d] = dydz * acc.x;
}

// project_sh (tools/FFT_sph.f90:247-279): a_lm = dy dz sum_jk w_jk f conj(Y_lm) sin(theta_j).
// Y_lm = (norm P_lm)(theta_j) (cos m phi_k, sin m phi_k); Y_l,-m = (-1)^m conj(Y_lm).
// One block per (l, m, detector), m on either side of zero in turn of l: the
// (L + 1)^2 pairs with |m| <= l, none of them empty; then, when `out` is given,
// three blocks per detector for the fluxes, which read the same shells.
__global__ void shell_reduce_kernel(const double2* shells, const int* active, int L, int Ny, int Nz,
                                    const double* __restrict__ normP, const double* __restrict__ cosm,
                                    const double* __restrict__ sinm, const double* __restrict__ sint, double dydz,
                                    double2* alm, double* out) {
  pdl_wait();
  const int d = blockIdx.y;
  if (!active[d]) return;
  int b = blockIdx.x;
  if (alm) {
    if (b >= (L + 1) * (L + 1)) {
      flux_block(shells, b - (L + 1) * (L + 1), d, Ny, Nz, dydz, out);
      return;
    }
  } else {
    flux_block(shells, b, d, Ny, Nz, dydz, out);
    return;
  }
  int l = (int)sqrtf((float)b);
  while (l * l > b) --l;
  while ((l + 1) * (l + 1) <= b) ++l;
  const int m = b - l * l - l, mi = m + L;
  const int am = m < 0 ? -m : m;
  const double sgn = (am & 1) ? -1.0 : 1.0;
  const double* P = normP + ((long long)l * (L + 1) + am) * Ny;
  const double* cm = cosm + (long long)am * Nz;
  const double* sm = sinm + (long long)am * Nz;
  const double2* f = shells + ((long long)d * 4) * Ny * Nz;
  double2 acc = c2(0.0, 0.0);
  for (int t = threadIdx.x; t < Ny * Nz; t += blockDim.x) {
    const int jv = t % Ny, kv = t / Ny;
    const double np = P[jv];
    double2 y = c2(np * cm[kv], np * sm[kv]);
    if (m < 0) y = c2(sgn * y.x, sgn * -y.y);
    const double2 a = f[t];
    const double2 cy = c2(y.x, -y.y);
    const double2 fy = c2(a.x * cy.x - a.y * cy.y, a.x * cy.y + a.y * cy.x);
    const double s = sint[jv];
    const double2 fun = c2(fy.x * s, fy.y * s);
    acc = cadd(acc, rmul(trap_w(jv, kv, Ny, Nz), fun));
  }
  acc = block_sum2(acc);
  if (threadIdx.x == 0) alm[(long long)l + (L + 1) * ((long long)mi + (2 * L + 1) * d)] = rmul(dydz, acc);
}

void launch_shell_reduce(const double2* shells, const int* active, int n_det, int L, int Ny, int Nz,
                         const double* normP, const double* cosm, const double* sinm, const double* sint, double dydz,
                         double2* alm, double* flux, cudaStream_t st) {
  const int nb = (alm ? (L + 1) * (L + 1) : 0) + (flux ? 3 : 0);
  launch_pdl(shell_reduce_kernel, dim3(nb, n_det), 256, 0, st, shells, active, L, Ny, Nz, normP, cosm, sinm, sint, dydz,
             alm, flux);
}

}  // namespace kg
