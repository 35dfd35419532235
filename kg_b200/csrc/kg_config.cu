// kg_config.cu -- the configured method (scheme 1): fourth-order centred
// differences, sixth-order Kreiss-Oliger dissipation and a Sommerfeld outer
// boundary, with RK4.  The reference wires only second-order operators (its
// fourth-order x stencil, first_derivative_x_4 in
// tools/finite_differences.f90:124-154, is real-only and never called), so this
// method is defined here and by the oracle's restatement of it, which this code
// matches to 1e-13 (multiply-adds are contracted, and the phi operators are formed
// as differences and sums of the stored variables, weighted by the metric and
// scaled afterwards; see cfg_phi):
//   * D4 f = (f(-2) - 8 f(-1) + 8 f(+1) - f(+2)) / (12 h) in r, theta and phi;
//     in r the one-sided closures of first_derivative_x_4 on the first and last
//     two stored planes; theta on the interior rows (the +-2 rows of the first
//     and last interior rows are ghost rows); phi periodic over the Nz-1
//     distinct planes.  The shift advection term uses D4 as well, and d_r beta
//     is the D4 derivative of beta^r.
//   * + eps / (64 h) (f(-3) - 6 f(-2) + 15 f(-1) - 20 f + 15 f(+1) - 6 f(+2) + f(+3))
//     per direction on all five variables (r planes 3..N-3 only).
//   * the outermost r plane obeys d_t u = -(d_r u + u / r) (Sommerfeld); the
//     innermost planes (inside the horizon) evolve with the one-sided closures.
//   * the theta ghost rows and the duplicated phi planes are not computed; they are
//     refilled after every stage: the phi planes first, then the theta ghost
//     rows from the interior rows at phi + pi with psi_2 negated (the parity of
//     d_theta of a smooth function on the sphere); the theta flux
//     alpha sqrt(gamma) gamma^thth psi_2 takes the sign of sin(theta), negative
//     on the ghost rows where the table holds |sqrt(gamma)|.
// Divisions by sqrt(gamma) and RK4's 1/6 use the correctly rounded reciprocal
// with one Markstein correction (the IEEE quotient for dividends above about
// 2^-1000 in magnitude).
#include <cuda.h>
#include <cuda_runtime.h>
#include "kg_device.cuh"
#include "kg_internal.h"
#include "kg_tma_ops.cuh"

namespace kg {
using namespace tmaops;
namespace {

struct CfgArgs {
  Grid g;
  Metric m;
  const double* dxb4;  // D4 d_r beta^r, [jj][ii] with pitch PI
  const double* rsg;   // 1 / sqrt(gamma), host-rounded, same layout
  const double2* in;   // stage input (5 variables, stride g.fs)
  const double2* base; // u^n
  double2* acc;
  double2* out;
  double rr, rt, rp;   // 1 / (12 h) per direction
  double kr, kt, kp;   // eps / (64 h) per direction
  double rN;           // r of the outermost stored plane
  int* err;            // set when a bounded wait runs out
};

// plane d steps from plane k (1 <= k <= Nz-1) over the Nz-1 distinct planes 1..Nz-1;
// |d| <= 4 <= Nz-1, so one wrap at most
__device__ __forceinline__ int kper(const Grid& g, int k, int d) {
  const int M = g.Nzm1;
  int kk = k - 1 + d;
  if (kk < 0) kk += M;
  if (kk >= M) kk -= M;
  return kk + 1;
}

// first_derivative_x_4 closures and centred stencil along r of a point function
template <class F>
__device__ __forceinline__ double2 d4r(const Grid& g, const F& f, int ii, double res) {
  const int n = g.NI - 1;
  double2 r;
  if (ii == 0)
    r = csub(cadd(csub(cadd(rmul(-25.0, f(0)), rmul(48.0, f(1))), rmul(36.0, f(2))), rmul(16.0, f(3))),
             rmul(3.0, f(4)));
  else if (ii == 1)
    r = cadd(csub(cadd(csub(rmul(-3.0, f(0)), rmul(10.0, f(1))), rmul(18.0, f(2))), rmul(6.0, f(3))),
             rmul(1.0, f(4)));
  else if (ii == n - 1)
    r = csub(cadd(csub(cadd(rmul(3.0, f(n)), rmul(10.0, f(n - 1))), rmul(18.0, f(n - 2))), rmul(6.0, f(n - 3))),
             rmul(1.0, f(n - 4)));
  else if (ii == n)
    r = cadd(csub(cadd(csub(rmul(25.0, f(n)), rmul(48.0, f(n - 1))), rmul(36.0, f(n - 2))), rmul(16.0, f(n - 3))),
             rmul(3.0, f(n - 4)));
  else
    r = csub(cadd(csub(f(ii - 2), rmul(8.0, f(ii - 1))), rmul(8.0, f(ii + 1))), f(ii + 2));
  return c2(r.x * res, r.y * res);
}
// what a point takes from the planes k+-1..3 of its own column: the dissipation's
// neighbours, and the fourth-order differences (times 12 h) that psi_3 and Pi need
struct Phi {
  double2 ko[5];
  double2 e;  // of alpha Pi + beta psi_1
  double2 f;  // of gamma^rphi psi_1 + gamma^phiphi psi_3
};
template <class PF>
__device__ __forceinline__ Phi cfg_phi(const CfgArgs& a, int q, const PF& P) {
  const Metric& M = a.m;
  Phi w;
  double2 d[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const double2 m3 = P(v, -3), m2 = P(v, -2), m1 = P(v, -1), p1 = P(v, 1), p2 = P(v, 2), p3 = P(v, 3);
    w.ko[v] = cadd(csub(cadd(m3, p3), rmul(6.0, cadd(m2, p2))), rmul(15.0, cadd(m1, p1)));
    d[v] = csub(csub(m2, p2), rmul(8.0, csub(m1, p1)));
  }
  w.e = cadd(rmul(ldm(M.alpha, q), d[4]), rmul(ldm(M.beta, q), d[1]));
  w.f = cadd(rmul(ldm(M.grp, q), d[1]), rmul(ldm(M.gpp, q), d[3]));
  return w;
}
__device__ __forceinline__ double2 d4c(double2 m2, double2 m1, double2 p1, double2 p2, double res) {
  const double2 r = csub(cadd(csub(m2, rmul(8.0, m1)), rmul(8.0, p1)), p2);
  return c2(r.x * res, r.y * res);
}
__device__ __forceinline__ double2 ko6(double2 m3, double2 m2, double2 m1, double2 c0, double2 p1, double2 p2,
                                       double2 p3) {
  return cadd(csub(cadd(csub(cadd(csub(m3, rmul(6.0, m2)), rmul(15.0, m1)), rmul(20.0, c0)), rmul(15.0, p1)),
                   rmul(6.0, p2)),
              p3);
}
__device__ __forceinline__ double2 cdiv(double2 a, double s) { return c2(a.x / s, a.y / s); }
// a / b from the correctly rounded reciprocal rb and one Markstein correction
// (q = a rb, r = a - q b, q + r rb): the IEEE quotient for dividends above about
// 2^-1000 in magnitude, at three operations instead of a division sequence
__device__ __forceinline__ double qdiv(double a, double b, double rb) {
  const double q = a * rb;
  const double r = __fma_rn(-q, b, a);
  return __fma_rn(r, rb, q);
}
__device__ __forceinline__ double2 cqdiv(double2 a, double b, double rb) { return c2(qdiv(a.x, b, rb), qdiv(a.y, b, rb)); }
constexpr double kSixth = 1.0 / 6.0;

// RHS and RK4 combination at one interior point (ii, jj, k): rows 3..NJ-4, planes
// 1..Nz-1 (the ghost fill behind every stage writes the others).  S(v, i, j) returns
// variable v of the stage input at (i, j) on plane k, w holds what the point's own
// column gives on the planes around it (cfg_phi, whose P(v, d) is the value d planes
// away); the two kernels below differ only in where S and P read from, so they
// produce the same bits.
template <int KIND, class SF>
__device__ __forceinline__ void cfg_point(const CfgArgs& a, int ii, int jj, int k, const SF& S, const Phi& w) {
  const Grid& g = a.g;
  const Metric& M = a.m;
  const long long p = off3(g, ii, jj, k);
  const int q = off2(g, ii, jj);
  double2 r[5];
  const int n = g.NI - 1;
  if (ii == n) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      auto f = [&](int i2) { return S(v, i2, jj); };
      r[v] = cneg(cadd(d4r(g, f, ii, a.rr), cdiv(S(v, ii, jj), a.rN)));
    }
  } else {
    const double al = ldm(M.alpha, q), b1 = ldm(M.beta, q), sg = ldm(M.sqrtg, q), dxb = ldm(a.dxb4, q);
    // alpha Pi + beta psi_1 on this plane
    auto ES = [&](int i2, int j2) {
      const int q2 = off2(g, i2, j2);
      return cadd(rmul(ldm(M.alpha, q2), S(4, i2, j2)), rmul(ldm(M.beta, q2), S(1, i2, j2)));
    };
    // sqrt(gamma) carries the sign of sin(theta) through the pole: negative on the ghost rows
    auto H = [&](int j2) {
      const double2 h = rmul(ldm(M.asg_gtt, off2(g, ii, j2)), S(2, ii, j2));
      return (j2 <= 2 || j2 >= g.NJ - 3) ? cneg(h) : h;
    };
    const double2 pi = S(4, ii, jj), ps1 = S(1, ii, jj);
    r[0] = cadd(rmul(al, pi), rmul(b1, ps1));
    {
      auto fA = [&](int i2) { return rmul(ldm(M.alpha, off2(g, i2, jj)), S(4, i2, jj)); };
      auto fP = [&](int i2) { return S(1, i2, jj); };
      r[1] = cadd(cadd(d4r(g, fA, ii, a.rr), rmul(b1, d4r(g, fP, ii, a.rr))), rmul(dxb, ps1));
    }
    r[2] = d4c(ES(ii, jj - 2), ES(ii, jj - 1), ES(ii, jj + 1), ES(ii, jj + 2), a.rt);
    r[3] = rmul(a.rp, w.e);
    {
      auto fG = [&](int i2) {
        const int q2 = off2(g, i2, jj);
        return rmul(ldm(M.asg, q2), cadd(rmul(ldm(M.grr, q2), S(1, i2, jj)), rmul(ldm(M.grp, q2), S(3, i2, jj))));
      };
      auto fQ = [&](int i2) {
        const double2 x = S(4, i2, jj);
        const double s2 = ldm(M.sqrtg, off2(g, i2, jj));
        return c2(x.x * s2, x.y * s2);
      };
      const double rs = ldm(a.rsg, q);
      const double2 t1 = cqdiv(d4r(g, fG, ii, a.rr), sg, rs);
      const double2 t2 = cqdiv(d4c(H(jj - 2), H(jj - 1), H(jj + 1), H(jj + 2), a.rt), sg, rs);
      const double2 t3 = cqdiv(rmul(a.rp, rmul(ldm(M.asg, q), w.f)), sg, rs);
      const double2 t4 = c2(pi.x * dxb, pi.y * dxb);
      const double2 t5 = cqdiv(rmul(b1, d4r(g, fQ, ii, a.rr)), sg, rs);
      const double2 t6 = rmul(ldm(M.am2, q), S(0, ii, jj));
      r[4] = csub(cadd(cadd(cadd(cadd(t1, t2), t3), t4), t5), t6);
    }
    const bool kor = ii >= 3 && ii <= n - 3;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      double2 s = r[v];
      if (kor)
        s = cadd(s, rmul(a.kr, ko6(S(v, ii - 3, jj), S(v, ii - 2, jj), S(v, ii - 1, jj), S(v, ii, jj),
                                   S(v, ii + 1, jj), S(v, ii + 2, jj), S(v, ii + 3, jj))));
      s = cadd(s, rmul(a.kt, ko6(S(v, ii, jj - 3), S(v, ii, jj - 2), S(v, ii, jj - 1), S(v, ii, jj),
                                 S(v, ii, jj + 1), S(v, ii, jj + 2), S(v, ii, jj + 3))));
      s = cadd(s, rmul(a.kp, csub(w.ko[v], rmul(20.0, S(v, ii, jj)))));
      r[v] = s;
    }
  }
  // RK4 combination, as the reference's k1..k4 form (MoL/lines_method_lib.f90:411-474)
  const double dt = g.dt;
  // the operands of all variables are requested ahead of the first store
  double2 bv[5], sv[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    bv[v] = lds(a.base, (long long)v * g.fs + p);
    if (KIND != ST_RK4_1) sv[v] = lds(a.acc, (long long)v * g.fs + p);
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const long long o = (long long)v * g.fs + p;
    const double2 b = bv[v];
    const double2 kk = c2(r[v].x * dt, r[v].y * dt);
    double2 res;
    if (KIND == ST_RK4_1) {
      a.acc[o] = kk;
      res = cadd(b, rmul(0.50, kk));
    } else if (KIND == ST_RK4_2) {
      a.acc[o] = cadd(sv[v], rmul(2.0, kk));
      res = cadd(b, rmul(0.50, kk));
    } else if (KIND == ST_RK4_3) {
      a.acc[o] = cadd(sv[v], rmul(2.0, kk));
      res = cadd(b, kk);
    } else {
      res = cadd(b, cqdiv(cadd(sv[v], kk), 6.0, kSixth));
    }
    a.out[o] = res;
  }
}

// One thread per stored point; every neighbour through the read-only cache.
template <int KIND>
__global__ void __launch_bounds__(128) cfg_stage_kernel(CfgArgs a) {
  const Grid& g = a.g;
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  const int jj = 3 + blockIdx.y;
  const int k = 1 + blockIdx.z;
  if (ii >= g.NI) return;
  const double2* U = a.in;
  auto S = [&](int v, int i2, int j2) { return ldf(U + (long long)v * g.fs, off3(g, i2, j2, k)); };
  auto P = [&](int v, int d) { return ldf(U + (long long)v * g.fs, off3(g, ii, jj, kper(g, k, d))); };
  cfg_point<KIND>(a, ii, jj, k, S, cfg_phi(a, off2(g, ii, jj), P));
}

// Tiled form: a CTA owns a 32 x 8 tile of (r, theta) columns of the interior rows
// and marches through a chunk of the planes 1..Nz-1.  The plane being updated
// arrives in shared memory with a +-4 r and +-3 theta halo (every same-plane
// neighbour the fourth-order differences, the r closures and the sixth-order
// dissipation touch), double buffered: one TMA box of all five variables brings
// the next plane's tile while this plane is computed.  The phi neighbours (planes
// k+-1..3 of the thread's own column) are plain loads that come from L2 on every
// plane; cfg_phi reads them ahead of the wait for the tile, a variable's six
// together, and keeps seven sums of them.  What bounds it is the chain of one
// plane's loads and fifteen stencils at 16 warps per SM.  256 x 33 x 65, event-timed
// us of stages 1 to 4: with cp.async tiles of every row and the neighbours loaded
// where the formulas name them 142, 171, 169, 166; now 86, 94, 94, 90 (an RK4 step
// with its fills 0.612 / 0.365 ms).  Slower: the point-wise operands prefetched into
// L2 a plane ahead (20 steps 7.99 ms for 7.92), u^n staged in shared memory (9.2 ms,
// with 8 KB of L1 left), and the neighbours in a rolling register window (255
// registers per thread, one CTA per SM: half the speed).
constexpr int CTI = 32, CTJ = 8, CRH = 4, CTH = 3;
constexpr int CW = CTI + 2 * CRH, CH = CTJ + 2 * CTH, CT_N = CW * CH;
constexpr size_t CFG_TILE_BYTES = (size_t)5 * CT_N * sizeof(double2);

template <int KIND>
__global__ void __launch_bounds__(CTI * CTJ, 2)
    cfg_march_kernel(const __grid_constant__ CUtensorMap tm, CfgArgs a, int kchunk) {
  extern __shared__ __align__(128) unsigned char cfg_smem[];
  double2* tiles;
  {
    const uint32_t b = saddr(cfg_smem);
    tiles = reinterpret_cast<double2*>(cfg_smem + ((128u - (b & 127u)) & 127u));
  }
  __shared__ uint64_t bars[2];
  const Grid& g = a.g;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * CTI + tx;
  const int ii0 = blockIdx.x * CTI, jj0 = 3 + blockIdx.y * CTJ;
  const int ii = ii0 + tx, jj = jj0 + ty;
  const bool act = ii < g.NI && jj < g.NJ - 3;
  const int k0 = 1 + blockIdx.z * kchunk, k1 = min(k0 + kchunk, g.Nz);
  const double2* col = a.in + (act ? off3(g, ii, jj, 0) : 0);
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  auto load = [&](int k, int buf) {  // the box starts at most 4 columns before the array, where it reads zeros
    mbar_expect_tx(&bars[buf], (uint32_t)CFG_TILE_BYTES);
    tma_load_4d(tiles + (size_t)buf * 5 * CT_N, &tm, 2 * (ii0 - CRH), jj0 - CTH, k, 0, &bars[buf]);
  };
  if (tid == 0) load(k0, 0);
  int timed_out = 0;
  bool failed = false;
  int last = k0;  // the plane of the newest copy
  for (int k = k0; k < k1 && !failed; ++k) {
    const int buf = (k - k0) & 1;
    if (k + 1 < k1) {
      if (tid == 0) load(k + 1, buf ^ 1);  // that buffer was last read before the barrier of the plane before
      last = k + 1;
    }
    auto P = [&](int v, int d) { return lds(col + (long long)v * g.fs, (long long)kper(g, k, d) * g.plane); };
    Phi w = {};
    if (act) w = cfg_phi(a, off2(g, ii, jj), P);
    if (!mbar_wait_bounded(&bars[buf], (uint32_t)((k - k0) >> 1) & 1u)) timed_out = 1;
    if (act && !timed_out) {
      // every same-plane neighbour lies inside the halo tile
      const double2* T = tiles + (size_t)buf * 5 * CT_N + (ty + CTH) * CW + (tx + CRH);
      auto S = [&](int v, int i2, int j2) { return T[v * CT_N + (j2 - jj) * CW + (i2 - ii)]; };
      cfg_point<KIND>(a, ii, jj, k, S, w);
    }
    failed = __syncthreads_or(timed_out) != 0;
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(a.err, 1);
      // the newest copy into either buffer lands before the CTA's shared memory is released (bounded)
      for (int q = last; q >= k0 && q > last - 2; --q)
        (void)mbar_wait_bounded(&bars[(q - k0) & 1], (uint32_t)((q - k0) >> 1) & 1u);
    }
    __syncthreads();
  }
}

// The method's fill: phi planes 0 <- Nz-1 and Nz <- 1, then the theta ghost rows
// from the interior rows at phi + pi, psi_2 negated.  One launch, a block per row:
// a ghost row whose partner is plane 0 reads plane Nz-1, its source, so no row that
// is read is written (256 x 33 x 65, event-timed us in two launches and in one: 20.6 /
// 8.8).
__global__ void cfg_ghost_kernel(Grid g, double2* u) {
  pdl_wait();
  const int nz = 2 * (g.NJ - 6);  // interior rows of the two planes
  int jd, kd, js, ks;
  bool ghost = false;
  if ((int)blockIdx.x < nz) {
    jd = js = 3 + blockIdx.x % (g.NJ - 6);
    const bool last = (int)blockIdx.x >= g.NJ - 6;
    kd = last ? g.Nz : 0;
    ks = last ? 1 : g.Nz - 1;
  } else {
    const int q = blockIdx.x - nz, r = q % 6;
    ghost = true;
    kd = q / 6;
    jd = r < 3 ? r : g.NJ - 6 + r;
    js = jd <= 2 ? 5 - jd : 2 * g.NJ - 7 - jd;
    ks = ktarget(g, kd);
    if (ks == 0) ks = g.Nz - 1;
  }
  for (int ii = threadIdx.x; ii < g.NI; ii += blockDim.x) {
    double2 s[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) s[v] = u[(long long)v * g.fs + off3(g, ii, js, ks)];
    if (ghost) s[2] = rmul(-1.0, s[2]);
#pragma unroll
    for (int v = 0; v < 5; ++v) u[(long long)v * g.fs + off3(g, ii, jd, kd)] = s[v];
  }
}

typedef CUresult (*EncodeTiledFnC)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// the stage input as (doubles along r, theta rows, phi planes, variables), boxes of
// one plane's halo tile
bool cfg_encode(CUtensorMap* tm, const Grid& g, const double2* base) {
  static EncodeTiledFnC fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFnC)p;
    if (!fn) return false;
  }
  cuuint64_t dims[4] = {(cuuint64_t)(2 * g.PI), (cuuint64_t)g.NJ, (cuuint64_t)g.NK, 5};
  cuuint64_t strides[3] = {(cuuint64_t)g.PI * 16, (cuuint64_t)g.plane * 16, (cuuint64_t)g.fs * 16};
  cuuint32_t box[4] = {2 * CW, CH, 1, 5};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void*)base, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int KIND>
int cfg_march_launch(const CfgArgs& a, cudaStream_t st) {
  constexpr int SMEM = 2 * (int)CFG_TILE_BYTES + 128;
  if (!allow_smem<cfg_march_kernel<KIND>>(SMEM)) return -1;
  const Grid& g = a.g;
  CUtensorMap tm;
  if (!cfg_encode(&tm, g, a.in)) return -1;
  const int tx = (g.NI + CTI - 1) / CTI, ty = (g.NJ - 6 + CTJ - 1) / CTJ, planes = g.Nz - 1;
  const int kchunk = phi_chunk(planes, (long long)tx * ty, 148 * 2, 32);
  return launch_pdl_or_refuse(cfg_march_kernel<KIND>, dim3(tx, ty, (planes + kchunk - 1) / kchunk), dim3(CTI, CTJ, 1),
                              SMEM, st, tm, a, kchunk);
}

}  // namespace

int launch_stage_cfg(int kind, const StageLaunch& L, const double* dxbeta4, const double* rsg, const double coef[6],
                     double rN, int tiled, int* err, cudaStream_t st) {
  CfgArgs a;
  a.g = L.g;
  a.m = L.m;
  a.dxb4 = dxbeta4;
  a.rsg = rsg;
  a.in = L.in[0];
  a.base = L.base;
  a.acc = L.acc;
  a.out = L.out;
  a.rr = coef[0];
  a.rt = coef[1];
  a.rp = coef[2];
  a.kr = coef[3];
  a.kt = coef[4];
  a.kp = coef[5];
  a.rN = rN;
  a.err = err;
  if (tiled) {  // without tensor maps: one thread per point
    switch (kind) {
      case ST_RK4_1: if (cfg_march_launch<ST_RK4_1>(a, st) == 0) return 0; break;
      case ST_RK4_2: if (cfg_march_launch<ST_RK4_2>(a, st) == 0) return 0; break;
      case ST_RK4_3: if (cfg_march_launch<ST_RK4_3>(a, st) == 0) return 0; break;
      case ST_RK4_4: if (cfg_march_launch<ST_RK4_4>(a, st) == 0) return 0; break;
      default: return -1;
    }
  }
  dim3 grid((L.g.NI + 127) / 128, L.g.NJ - 6, L.g.Nz - 1);
  switch (kind) {
    case ST_RK4_1: cfg_stage_kernel<ST_RK4_1><<<grid, 128, 0, st>>>(a); return 0;
    case ST_RK4_2: cfg_stage_kernel<ST_RK4_2><<<grid, 128, 0, st>>>(a); return 0;
    case ST_RK4_3: cfg_stage_kernel<ST_RK4_3><<<grid, 128, 0, st>>>(a); return 0;
    case ST_RK4_4: cfg_stage_kernel<ST_RK4_4><<<grid, 128, 0, st>>>(a); return 0;
    default: return -1;
  }
}

void launch_ghost_fill_cfg(const Grid& g, double2* u, cudaStream_t st) {
  const int nt = g.NI >= 256 ? 256 : (g.NI + 31) / 32 * 32;
  launch_pdl(cfg_ghost_kernel, 2 * (g.NJ - 6) + 6 * g.NK, nt, 0, st, g, u);
}

}  // namespace kg
