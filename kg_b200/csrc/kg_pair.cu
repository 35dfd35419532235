// kg_pair.cu -- two RK4 stages in one pass over memory.
//
// An RK4 step (MoL/lines_method_lib.f90:411-474) run as four stage kernels moves
// 1360 B per point: every stage output goes to HBM and comes back through the
// next stage's stencil.  Here stages 1 and 2, and stages 3 and 4, are one kernel
// each, with the output of the first of the two kept on the chip:
//   pair 0 (stages 1, 2):  X = u^n:  k1 = dt rhs(X), Y = u + k1/2, k2 = dt rhs(Y);
//                          writes the sum k1 + 2 k2 and u + k2/2   (80 in, 160 out)
//   pair 1 (stages 3, 4):  X = pair 0's u + k2/2: k3 = dt rhs(X), Y = u + k3,
//                          k4 = dt rhs(Y); writes u^{n+1}          (240 in, 80 out)
// which is 560 B per point and step.  u^{n+1} goes to another buffer than u^n,
// since neighbouring tiles form Y on their halo from u^n.
//
// Work layout.  A CTA owns 28 r columns x TJ theta rows and marches through a
// chunk of phi planes.  It forms Y on a region one row taller on either side and
// 32 columns wide: warp w stands at row j0 - 1 + w, lane L at column i0 - 2 + L,
// so lanes 2..29 of warps 1..TJ are the tile's own points.  Per plane P[s]:
//   * X arrives by TMA (one box of all five variables, +-2 columns and +-1 row
//     around the region) in a 3-deep ring with one "full" mbarrier per slot;
//   * every warp forms Y of P[s] at its region points and puts psi1 and the five
//     products of Y with the metric that neighbours difference into a
//     double-buffered plane in shared memory, each formed once by its own point;
//   * the own points form the second right-hand side of P[s-1] from that plane's
//     products, with the phi neighbours' arguments in registers.  The first
//     increment (pair 0) or the increment sum (pair 1) of P[s-1] waits in shared
//     memory, and so does u in pair 0; pair 1 reads u again;
//   * one block barrier orders the Y planes and frees X's slot.
// The ghost values of Y that the reference's boundary() would put in between:
//   r: the excision extrapolation and the outer copy (or hold) come from the lanes
//     beside by shuffles (the region of a tile at an end holds them);
//   theta: the ghost row beside the first and last interior row is Y at that row
//     on the plane half a turn away.  launch_pole_rows forms Y on those two rows
//     beforehand and the region row outside the poles is read from its buffer;
//   phi: the plane before 1 is Nz - 1 and the one after Nz - 1 is 1: the planes are
//     taken cyclically.  That equals the reference's seam planes 0 and Nz when
//     the state holds plane 0 = plane Nz - 1 and plane Nz = plane 1, which every
//     ghost fill leaves; the caller runs a state that no fill has seen yet through
//     the four stage kernels.
// Every value is formed with the operations of the stage kernels (kg_tma.cu) in
// their order, so the results are the same bits.
//
// What bounds it: not memory (30 % of the HBM rate) but the latency of the two
// dependent right-hand sides at 10 warps per SM, all that the X ring, the Y planes,
// the parked values and the metric tile leave room for (FP64 pipe 33 % busy, then
// LDS latency and the barrier).  Event-timed us, the two stage kernels, which store
// their ghost values, and the pair, whose fill and pole rows take 32 us each (13 on
// the second grid) on top: 1024 x 65 x 129 1036 / 693 and 1116 / 868, 301 x 46 x 90
// 188 / 137 and 205 / 174.  Why this split (1024 x 65 x 129, pair 0 / pair 1 of the variant against
// the same form otherwise): tiles of 4 rows with two CTAs per SM 809 / 1099 for 787 /
// 990; products formed by each neighbour and the sum in registers 787 / 990 for 697 /
// 867; tiles of 10 rows 712 / 1033, the march in copies per warp role 781 / 993 and
// the second right-hand side ahead of the Y stores 736 / 1039 for 686 / 864; ghost
// values stored by the pairs 1938 us a step for 1658.
#include <cuda.h>
#include <cuda_runtime.h>
#include "kg_device.cuh"
#include "kg_internal.h"
#include "kg_tma_ops.cuh"

namespace kg {
using namespace tmaops;
namespace {

constexpr int PO = 28;      // own r columns of a tile
constexpr int TJ = 8;       // and theta rows
constexpr int PW = 36;      // ring and metric tile width: the 32 region columns +- 2
constexpr int PST = 3;      // ring depth
enum { PT_AL = 0, PT_BE, PT_A, PT_GRR, PT_GRP, PT_SG, PT_HT, PT_COUNT };
// what a Y plane holds: psi1 and the products with the metric that neighbours
// difference, each formed once by its own point
enum { Y_P1 = 0, Y_AP, Y_E, Y_G, Y_H, Y_Q, Y_COUNT };

// Shared memory of a tile.  Of the Y planes and the metric tables
// only E, H and alpha, beta, (alpha sqrtg) gamma^thth are read beyond the own (the
// region's) rows.
struct PGeom {
  static constexpr int WARPS = TJ + 2, ROWS = TJ + 4;
  static constexpr int FULL = ROWS * PW, PART = WARPS * PW;  // complex values per variable and plane
  static constexpr uint32_t TX_B = 5 * FULL * 16;            // bytes of a plane's box
  static constexpr int SLOT = (TX_B + 127) / 128 * 128;
  static constexpr int Y_WIDE = WARPS * 32, Y_OWN = TJ * 32;  // points of a Y array: region rows, own rows
  // a Y plane: E and H on the region's rows, then the other four on the own rows
  static __host__ __device__ constexpr int y_at(int w) {
    return w == Y_E ? 0 : w == Y_H ? Y_WIDE : 2 * Y_WIDE + (w == Y_P1 ? 0 : w == Y_AP ? 1 : w == Y_G ? 2 : 3) * Y_OWN;
  }
  static constexpr int Y_PLANE = 2 * Y_WIDE + 4 * Y_OWN;
  static constexpr int PARK_N = TJ * 32;  // own points, by thread
  // metric tables: alpha, beta, H factor with the row halo, the others on the region's rows
  static __host__ __device__ constexpr bool m_full(int t) { return t == PT_AL || t == PT_BE || t == PT_HT; }
  static __host__ __device__ constexpr int m_at(int t) {
    return t == PT_AL ? 0
         : t == PT_BE ? FULL
         : t == PT_HT ? 2 * FULL
                      : 3 * FULL + (t == PT_A ? 0 : t == PT_GRR ? 1 : t == PT_GRP ? 2 : 3) * PART;
  }
  static constexpr int M_ALL = 3 * FULL + 4 * PART;
  static constexpr size_t SMEM =
      (size_t)PST * SLOT + 2 * (size_t)Y_PLANE * 16 + (size_t)10 * PARK_N * 16 + (size_t)M_ALL * 8 + 64 + 128;
  static_assert(SMEM <= 227 * 1024, "one CTA per SM");
};

struct PairArgs {
  Grid g;
  Metric m;
  const double* rsg;
  const double2* base;  // u^n
  const double2* acc_in;
  double2* acc_out;
  double2* out;
  const double2* pole;  // Y at rows 3 and NJ-4: [side][variable][k][PI]
  int inflow;
  int kchunk;
  int* err;
};

template <bool B>
struct PBool {
  static constexpr bool value = B;
};
__device__ __forceinline__ double pdiv(double a, double b, double rb) {
  const double q = a * rb;
  const double r = __fma_rn(-q, b, a);
  return __fma_rn(r, rb, q);
}
__device__ __forceinline__ double2 pcdiv(double2 a, double b, double rb) {
  return c2(pdiv(a.x, b, rb), pdiv(a.y, b, rb));
}
__device__ __forceinline__ double2 shfl_c(double2 v, int lane) {
  return c2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
// plane k of the Nz - 1 distinct ones, k from -1 to Nz + 1
__device__ __forceinline__ int cyc(const Grid& g, int k) {
  if (k < 1) k += g.Nzm1;
  else if (k > g.Nzm1) k -= g.Nzm1;
  return k;
}

struct Own {  // metric at the thread's own point
  double al, be, dxb, sg, rs, am2, fa, fgrp, fgpp;
};
// phi-derivative arguments of the psi and Pi right-hand sides
__device__ __forceinline__ double2 arg_e(const Own& o, double2 ps1, double2 pi) {
  return cadd(rmul(o.al, pi), rmul(o.be, ps1));
}
template <int MK>
__device__ __forceinline__ double2 arg_f(const Own& o, double2 ps1, double2 ps3) {
  if (MK == MK_KS) return rmul(o.fa, cadd(rmul(o.fgrp, ps1), rmul(o.fgpp, ps3)));
  return rmul(o.fa, ps3);
}

// rhs_phi .. rhs_pi (MoL/lines_method_lib.f90:671-743) at the own point.  RF(v, dx,
// dy): the stencil input, MT(table, dx, dy): the metric, at an offset; phi: its
// first variable here; Ep .. Fn: the phi arguments on the planes beside.  FAST as
// in kg_tma.cu: all lanes take the centred and the forward upwind differences.
template <bool FAST, int MK, class RFT, class MTT>
__device__ __forceinline__ void pair_rhs(const Grid& g, const Own& o, int ii, const RFT& RF, const MTT& MT, double2 phi,
                                         double2 Ep, double2 En, double2 Fp, double2 Fn, double2 r[5]) {
  const int n = g.NI - 1;
  const double2 ps1 = RF(1, 0, 0), pi = RF(4, 0, 0);
  r[0] = cadd(rmul(o.al, pi), rmul(o.be, ps1));
  {
    auto aPi = [&](int dx) { return rmul(MT(PT_AL, dx, 0), RF(4, dx, 0)); };
    auto f1 = [&](int dx) { return RF(1, dx, 0); };
    double2 d;
    if (FAST) d = ctr(aPi(-1), aPi(1));
    else if (ii == 0) d = fwd3(aPi(0), aPi(1), aPi(2));
    else if (ii == n) d = bwd3(aPi(0), aPi(-1), aPi(-2));
    else d = ctr(aPi(-1), aPi(1));
    d = rmul(g.rdx, d);
    double2 av;
    if (FAST) av = fwd3(ps1, f1(1), f1(2));
    else if (ii <= 1) av = fwd3(ps1, f1(1), f1(2));
    else if (ii == n - 1) av = csub(f1(1), f1(-1));
    else if (ii == n) av = bwd3(ps1, f1(-1), f1(-2));
    else if (o.be > 0.0) av = fwd3(ps1, f1(1), f1(2));
    else if (o.be < 0.0) av = bwd3(ps1, f1(-1), f1(-2));
    else av = csub(f1(1), f1(-1));
    av = rmul(g.rdx, av);
    r[1] = cadd(cadd(d, rmul(o.be, av)), rmul(o.dxb, ps1));
  }
  {
    auto E = [&](int dy) { return cadd(rmul(MT(PT_AL, 0, dy), RF(4, 0, dy)), rmul(MT(PT_BE, 0, dy), RF(1, 0, dy))); };
    r[2] = rmul(g.rdy, ctr(E(-1), E(1)));
  }
  r[3] = rmul(g.rdz, ctr(Ep, En));
  {
    auto G1 = [&](int dx) {
      if (MK == MK_KS)
        return rmul(MT(PT_A, dx, 0),
                    cadd(rmul(MT(PT_GRR, dx, 0), RF(1, dx, 0)), rmul(MT(PT_GRP, dx, 0), RF(3, dx, 0))));
      return rmul(MT(PT_A, dx, 0), RF(1, dx, 0));
    };
    double2 d;
    if (FAST) d = ctr(G1(-1), G1(1));
    else if (ii == 0) d = fwd3(G1(0), G1(1), G1(2));
    else if (ii == n) d = bwd3(G1(0), G1(-1), G1(-2));
    else d = ctr(G1(-1), G1(1));
    const double2 r1 = pcdiv(rmul(g.rdx, d), o.sg, o.rs);
    auto H = [&](int dy) { return rmul(MT(PT_HT, 0, dy), RF(2, 0, dy)); };
    const double2 r2 = pcdiv(rmul(g.rdy, ctr(H(-1), H(1))), o.sg, o.rs);
    const double2 z = rmul(g.rdz, ctr(Fp, Fn));
    const double2 r3 = (MK == MK_KS) ? pcdiv(z, o.sg, o.rs) : z;
    const double2 r4 = rmul(o.dxb, pi);
    auto Q = [&](int dx) { return rmul(MT(PT_SG, dx, 0), RF(4, dx, 0)); };
    double2 av;
    if (FAST) av = fwd3(Q(0), Q(1), Q(2));
    else if (ii <= 1) av = fwd3(Q(0), Q(1), Q(2));
    else if (ii == n - 1) av = csub(Q(1), Q(-1));
    else if (ii == n) av = bwd3(Q(0), Q(-1), Q(-2));
    else if (o.be > 0.0) av = fwd3(Q(0), Q(1), Q(2));
    else if (o.be < 0.0) av = bwd3(Q(0), Q(-1), Q(-2));
    else av = csub(Q(1), Q(-1));
    av = rmul(g.rdx, av);
    const double2 r5 = pcdiv(rmul(o.be, av), o.sg, o.rs);
    const double2 r6 = rmul(o.am2, phi);
    r[4] = csub(cadd(cadd(cadd(cadd(r1, r2), r3), r4), r5), r6);
  }
}

// The same from a Y plane's products.  Y(w, dx, dy): product w at an offset; phi, pi:
// the own point's first and last variable.
template <bool FAST, class YT>
__device__ __forceinline__ void pair_rhs_y(const Grid& g, const Own& o, int ii, bool ks, const YT& Y, double2 phi,
                                           double2 pi, double2 Ep, double2 En, double2 Fp, double2 Fn, double2 r[5]) {
  const int n = g.NI - 1;
  auto dr = [&](int w) {  // centred, one-sided at the ends
    double2 d;
    if (FAST) d = ctr(Y(w, -1, 0), Y(w, 1, 0));
    else if (ii == 0) d = fwd3(Y(w, 0, 0), Y(w, 1, 0), Y(w, 2, 0));
    else if (ii == n) d = bwd3(Y(w, 0, 0), Y(w, -1, 0), Y(w, -2, 0));
    else d = ctr(Y(w, -1, 0), Y(w, 1, 0));
    return rmul(g.rdx, d);
  };
  auto ar = [&](int w) {  // upwind by the sign of beta^r
    double2 av;
    if (FAST || ii <= 1) av = fwd3(Y(w, 0, 0), Y(w, 1, 0), Y(w, 2, 0));
    else if (ii == n - 1) av = csub(Y(w, 1, 0), Y(w, -1, 0));
    else if (ii == n) av = bwd3(Y(w, 0, 0), Y(w, -1, 0), Y(w, -2, 0));
    else if (o.be > 0.0) av = fwd3(Y(w, 0, 0), Y(w, 1, 0), Y(w, 2, 0));
    else if (o.be < 0.0) av = bwd3(Y(w, 0, 0), Y(w, -1, 0), Y(w, -2, 0));
    else av = csub(Y(w, 1, 0), Y(w, -1, 0));
    return rmul(g.rdx, av);
  };
  r[0] = Y(Y_E, 0, 0);
  r[1] = cadd(cadd(dr(Y_AP), rmul(o.be, ar(Y_P1))), rmul(o.dxb, Y(Y_P1, 0, 0)));
  r[2] = rmul(g.rdy, ctr(Y(Y_E, 0, -1), Y(Y_E, 0, 1)));
  r[3] = rmul(g.rdz, ctr(Ep, En));
  const double2 r1 = pcdiv(dr(Y_G), o.sg, o.rs);
  const double2 r2 = pcdiv(rmul(g.rdy, ctr(Y(Y_H, 0, -1), Y(Y_H, 0, 1))), o.sg, o.rs);
  const double2 z = rmul(g.rdz, ctr(Fp, Fn));
  const double2 r3 = ks ? pcdiv(z, o.sg, o.rs) : z;
  const double2 r4 = rmul(o.dxb, pi);
  const double2 r5 = pcdiv(rmul(o.be, ar(Y_Q)), o.sg, o.rs);
  const double2 r6 = rmul(o.am2, phi);
  r[4] = csub(cadd(cadd(cadd(cadd(r1, r2), r3), r4), r5), r6);
}

}  // namespace

template <int PAIR, int MK>
__global__ void __launch_bounds__(PGeom::WARPS * 32, 1)
    rk4_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU,
                    const __grid_constant__ CUtensorMap tmA, PairArgs a) {
  using GT = PGeom;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* ring;
  {
    const uint32_t b = saddr(smem_raw);
    ring = smem_raw + ((128u - (b & 127u)) & 127u);
  }
  double2* ybuf = reinterpret_cast<double2*>(ring + (size_t)PST * GT::SLOT);  // 2 planes of products
  double2* park = ybuf + 2 * GT::Y_PLANE;  // increment sum and u at P[s-1], by own thread
  double* mt = reinterpret_cast<double*>(park + 10 * GT::PARK_N);
  uint64_t* bars = reinterpret_cast<uint64_t*>(mt + GT::M_ALL);
  const Grid& g = a.g;
  const Metric& M = a.m;
  const int lane = threadIdx.x, w = threadIdx.y, tid = w * 32 + lane;
  const int i0 = 1 + blockIdx.x * PO, j0 = 3 + blockIdx.y * TJ;
  const int ii = i0 - 2 + lane, jj = j0 - 1 + w;
  const int k0 = 1 + blockIdx.z * a.kchunk, k1 = min(k0 + a.kchunk, g.Nz);  // own planes [k0, k1)
  const int nX = k1 - k0 + 4;  // X on planes k0 - 2 .. k1 + 1; Y on X planes 1 .. nX - 2
  auto plane_of = [&](int t) { return cyc(g, k0 - 2 + t); };
  const bool vcol = ii >= 0 && ii < g.NI;
  const bool ghost_row = jj == 2 || jj == g.NJ - 3;      // Y from the pole rows
  const bool form = vcol && jj >= 3 && jj <= g.NJ - 4;   // Y formed here
  const bool own = w >= 1 && w <= TJ && lane >= 2 && lane < 2 + PO && jj <= g.NJ - 4 && ii <= g.NI - 2;

  if (tid == 0) {
    for (int s = 0; s < PST; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue = [&](int t) {
    uint64_t* b = &bars[t % PST];
    mbar_expect_tx(b, GT::TX_B);
    tma_load_4d(ring + (size_t)(t % PST) * GT::SLOT, &tmX, 2 * (i0 - 4), j0 - 2, plane_of(t), 0, b);
  };
  // the point-wise operands of a plane, pulled into L2 ahead of their loads
  auto prefetch = [&](int t) {
    if (PAIR == 0 || t > nX - 2) return;
    tma_prefetch_4d(&tmU, 2 * (i0 - 1), j0 - 1, plane_of(t), 0);
    if (t >= 2 && t <= nX - 3) tma_prefetch_4d(&tmA, 2 * i0, j0, plane_of(t), 0);
  };
  int nissued = 0;
  if (tid == 0) {
    pdl_wait();
    for (int t = 0; t < PST; ++t) issue(t);  // nX >= 5
    nissued = PST;
    prefetch(1);
    prefetch(2);
  }
  for (int t = tid; t < GT::FULL; t += GT::WARPS * 32) {
    const int row = t / PW, gi = i0 - 4 + t % PW, gj = j0 - 2 + row;
    const bool in = gi >= 0 && gi < g.NI && gj < g.NJ;
    const int q = in ? off2(g, gi, gj) : 0;
    mt[GT::m_at(PT_AL) + t] = in ? ldm(M.alpha, q) : 0.0;
    mt[GT::m_at(PT_BE) + t] = in ? ldm(M.beta, q) : 0.0;
    mt[GT::m_at(PT_HT) + t] = in ? ldm(M.asg_gtt, q) : 0.0;
    if (row >= 1 && row <= GT::WARPS) {
      const int u = t - PW;
      mt[GT::m_at(PT_A) + u] = in ? ldm(MK == MK_KS ? M.asg : M.asg_grr, q) : 0.0;
      mt[GT::m_at(PT_GRR) + u] = in ? ldm(M.grr, q) : 0.0;
      mt[GT::m_at(PT_GRP) + u] = in ? ldm(M.grp, q) : 0.0;
      mt[GT::m_at(PT_SG) + u] = in ? ldm(M.sqrtg, q) : 0.0;
    }
  }
  Own o = {0, 0, 0, 1, 1, 0, 0, 0, 0};
  if (vcol && jj < g.NJ) {
    const int q = off2(g, ii, jj);
    o.al = ldm(M.alpha, q);
    o.be = ldm(M.beta, q);
    o.dxb = ldm(M.dxbeta, q);
    o.sg = ldm(M.sqrtg, q);
    o.rs = ldm(a.rsg, q);
    o.am2 = ldm(M.am2, q);
    o.fa = ldm(MK == MK_KS ? M.asg : M.a_gpp, q);
    if (MK == MK_KS) {
      o.fgrp = ldm(M.grp, q);
      o.fgpp = ldm(M.gpp, q);
    }
  }
  __syncthreads();
  pdl_wait();  // ahead of this thread's own reads and writes of the state
  const long long fs = g.fs;
  const long long pcol = form ? off3(g, ii, jj, 0) : 0;
  const long long ps = (long long)g.NK * g.PI;  // variable stride of the pole rows
  const double2* pole = a.pole + (jj == 2 ? 0 : 5 * ps) + ii;
  // variable v of X's plane t at an offset from the own point
  auto XV = [&](int t, int v, int dx, int dy) -> double2 {
    return reinterpret_cast<const double2*>(ring + (size_t)(t % PST) * GT::SLOT)[v * GT::FULL + (w + 1 + dy) * PW +
                                                                                  lane + 2 + dx];
  };
  auto MT = [&](int which, int dx, int dy) {
    return mt[GT::m_at(which) + (w + (GT::m_full(which) ? 1 : 0) + dy) * PW + lane + 2 + dx];
  };
  const double dt = g.dt;

  int timed_out = 0;
  if (!mbar_wait_bounded(&bars[0], 0u) || !mbar_wait_bounded(&bars[1], 0u)) timed_out = 1;
  double2 Ep = c2(0, 0), Ec = Ep, Fp = Ep, Fc = Ep;          // X's phi arguments at P[s-1], P[s]
  double2 Yep = Ep, Yec = Ep, Yfp = Ep, Yfc = Ep;            // Y's at P[s-2], P[s-1]
  double2 yphi = Ep, ypi = Ep;                               // Y's phi and Pi at P[s-1]
  park += own ? (w - 1) * 32 + lane : 0;
  if (!timed_out) {
    Ep = arg_e(o, XV(0, 1, 0, 0), XV(0, 4, 0, 0));
    Fp = arg_f<MK>(o, XV(0, 1, 0, 0), XV(0, 3, 0, 0));
    Ec = arg_e(o, XV(1, 1, 0, 0), XV(1, 4, 0, 0));
    Fc = arg_f<MK>(o, XV(1, 1, 0, 0), XV(1, 3, 0, 0));
  }
  bool failed = __syncthreads_or(timed_out) != 0;
  const bool fast = __all_sync(0xffffffffu, form && ii >= 2 && ii <= g.NI - 3 && o.be > 0.0);

  auto march = [&](auto fastc) {
    constexpr bool FAST = decltype(fastc)::value;
    for (int s = 1; s <= nX - 2 && !failed; ++s) {
      // the barrier that ended the previous plane freed X's slot s - 1
      if (tid == 0) {
        if (s + 2 < nX) {
          issue(s + 2);
          nissued = s + 3;
        }
        prefetch(s + 2);
      }
      const int k = plane_of(s);
      const long long p = pcol + (long long)k * g.plane;
      if (!timed_out && !mbar_wait_bounded(&bars[(s + 1) % PST], ((s + 1) / PST) & 1)) timed_out = 1;
      double2 un[5], kn[5], y[5];
#pragma unroll
      for (int v = 0; v < 5; ++v) un[v] = kn[v] = y[v] = c2(0, 0);
      if (form && !timed_out) {
        auto RF = [&](int v, int dx, int dy) { return XV(s, v, dx, dy); };
        if (PAIR == 0) {
#pragma unroll
          for (int v = 0; v < 5; ++v) un[v] = RF(v, 0, 0);
        } else {
#pragma unroll
          for (int v = 0; v < 5; ++v) un[v] = lds(a.base, v * fs + p);
        }
        const double2 En = arg_e(o, XV(s + 1, 1, 0, 0), XV(s + 1, 4, 0, 0));
        const double2 Fn = arg_f<MK>(o, XV(s + 1, 1, 0, 0), XV(s + 1, 3, 0, 0));
        double2 r[5];
        pair_rhs<FAST, MK>(g, o, ii, RF, MT, RF(0, 0, 0), Ep, En, Fp, Fn, r);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          kn[v] = rmul(dt, r[v]);
          y[v] = cadd(un[v], PAIR == 0 ? rmul(0.50, kn[v]) : kn[v]);
        }
        Ep = Ec;
        Ec = En;
        Fp = Fc;
        Fc = Fn;
      }
      if (!FAST) {  // the x faces of Y (boundary_xL, boundary_xR)
        const int lx = 2 - i0;  // lane of column 0, when in the region
        if (lx + 2 >= 0) {      // only the first tile: i0 = 1, column 0 on lane 1
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const double2 e = cadd(csub(rmul(3.0, shfl_c(y[v], lx + 1)), rmul(3.0, shfl_c(y[v], lx + 2))),
                                   shfl_c(y[v], lx + 3));
            if (ii == 0) y[v] = e;
          }
        }
        const int ln = g.NI - 1 - (i0 - 2);  // lane of the outermost column
        if (ln < 32) {
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const double2 e = shfl_c(y[v], ln - 1);
            if (ii == g.NI - 1) y[v] = a.inflow ? un[v] : e;
          }
        }
      }
      if (ghost_row && vcol && !timed_out) {
        int kt = ktarget(g, k);
        if (kt == 0) kt = g.Nzm1;
        const double2* q = pole + (long long)kt * g.PI;
#pragma unroll
        for (int v = 1; v < 5; ++v) y[v] = lds(q, v * ps);
      }
      // stage 3's part of the sum, requested under the second right-hand side
      double2 an[5];
      const bool sum = PAIR == 1 && own && s >= 2 && s <= nX - 3;
#pragma unroll
      for (int v = 0; v < 5; ++v) an[v] = sum ? lds(a.acc_in, v * fs + p) : c2(0, 0);
      // Y's products with the metric at this point
      const double2 ap = rmul(o.al, y[4]);
      const double2 Yen = cadd(ap, rmul(o.be, y[1])), Yfn = arg_f<MK>(o, y[1], y[3]);
      double2* yb = ybuf + (size_t)(s & 1) * GT::Y_PLANE + tid;
      yb[GT::y_at(Y_E)] = Yen;
      yb[GT::y_at(Y_H)] = rmul(MT(PT_HT, 0, 0), y[2]);
      if (w >= 1 && w <= TJ) {
        yb -= 32;  // arrays of the own rows
        yb[GT::y_at(Y_P1)] = y[1];
        yb[GT::y_at(Y_AP)] = ap;
        yb[GT::y_at(Y_G)] =
            MK == MK_KS ? rmul(MT(PT_A, 0, 0), cadd(rmul(MT(PT_GRR, 0, 0), y[1]), rmul(MT(PT_GRP, 0, 0), y[3])))
                        : rmul(MT(PT_A, 0, 0), y[1]);
        yb[GT::y_at(Y_Q)] = rmul(o.sg, y[4]);
      }
      // the second right-hand side on the own points of P[s-1]
      if (own && s >= 3 && !timed_out) {
        const long long pm = pcol + (long long)plane_of(s - 1) * g.plane;
        const double2* ym = ybuf + (size_t)((s - 1) & 1) * GT::Y_PLANE + tid;
        auto Y = [&](int v, int dx, int dy) {
          return ym[GT::y_at(v) - (v == Y_E || v == Y_H ? 0 : 32) + dy * 32 + dx];
        };
        double2 r[5], ul[5];
        if (PAIR == 1)
#pragma unroll
          for (int v = 0; v < 5; ++v) ul[v] = lds(a.base, v * fs + pm);
        pair_rhs_y<FAST>(g, o, ii, MK == MK_KS, Y, yphi, ypi, Yep, Yen, Yfp, Yfn, r);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          const long long q = v * fs + pm;
          const double2 kk = rmul(dt, r[v]), ko = park[v * GT::PARK_N], uo = PAIR == 0 ? park[(5 + v) * GT::PARK_N] : ul[v];
          if (PAIR == 0) {
            a.acc_out[q] = cadd(ko, rmul(2.0, kk));
            a.out[q] = cadd(uo, rmul(0.50, kk));
          } else {
            a.out[q] = cadd(uo, pcdiv(cadd(ko, kk), 6.0, 1.0 / 6.0));
          }
        }
      }
      if (own) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          park[v * GT::PARK_N] = PAIR == 1 ? cadd(an[v], rmul(2.0, kn[v])) : kn[v];
          if (PAIR == 0) park[(5 + v) * GT::PARK_N] = un[v];
        }
      }
      yphi = y[0];
      ypi = y[4];
      Yep = Yec;
      Yec = Yen;
      Yfp = Yfc;
      Yfc = Yfn;
      // Y of P[s] is complete, Y of P[s-1] and X of P[s] have been read
      failed = __syncthreads_or(timed_out) != 0;
    }
  };
  if (fast) march(PBool<true>());
  else march(PBool<false>());
  if (failed) {
    if (tid == 0) {
      atomicExch(a.err, 1);
      // let the last copy issued into each ring slot land before the CTA's
      // shared memory is released (bounded as well)
      for (int s = 0; s < PST; ++s) {
        int tl = -1;
        for (int t = 0; t < nissued; ++t)
          if (t % PST == s) tl = t;
        if (tl >= 0) (void)mbar_wait_bounded(&bars[s], (tl / PST) & 1);
      }
    }
    __syncthreads();
  }
}

namespace {

typedef CUresult (*EncodeTiledFnP)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFnP encode_fn_p() {
  static EncodeTiledFnP fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFnP)p;
  }
  return fn;
}

// a 5-variable state as (doubles along r incl. row padding, theta rows, phi
// planes, variables), with a box of `cols` complex columns x `rows` rows of one
// plane of all variables
bool encode_state(CUtensorMap* tm, const Grid& g, const double2* base, int cols, int rows) {
  EncodeTiledFnP fn = encode_fn_p();
  if (!fn) return false;
  cuuint64_t dims[4] = {(cuuint64_t)(2 * g.PI), (cuuint64_t)g.NJ, (cuuint64_t)g.NK, 5};
  cuuint64_t strides[3] = {(cuuint64_t)g.PI * 16, (cuuint64_t)g.plane * 16, (cuuint64_t)g.fs * 16};
  cuuint32_t box[4] = {(cuuint32_t)(2 * cols), (cuuint32_t)rows, 1, 5};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void*)base, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int PAIR, int MK>
int pair_launch(const PairLaunch& L, const double* rsg, int* err, cudaStream_t st) {
  using GT = PGeom;
  if (!allow_smem<rk4_pair_kernel<PAIR, MK>>(GT::SMEM)) return -1;
  const Grid& g = L.g;
  CUtensorMap tmX, tmU, tmA;
  if (!encode_state(&tmX, g, L.X, PW, GT::ROWS) || !encode_state(&tmU, g, L.base, 32, GT::WARPS) ||
      !encode_state(&tmA, g, PAIR == 1 ? L.acc_in : L.base, PO, TJ))
    return -1;
  PairArgs a;
  a.g = g;
  a.m = L.m;
  a.rsg = rsg;
  a.base = L.base;
  a.acc_in = L.acc_in;
  a.acc_out = L.acc_out;
  a.out = L.out;
  a.pole = L.pole;
  a.inflow = L.inflow;
  a.err = err;
  dim3 grid((g.NI - 2 + PO - 1) / PO, (g.NJ - 6 + TJ - 1) / TJ, 1);
  a.kchunk = pair_chunk(g.Nz - 1, (long long)grid.x * grid.y);
  grid.z = (g.Nz - 1 + a.kchunk - 1) / a.kchunk;
  return launch_pdl_or_refuse(rk4_pair_kernel<PAIR, MK>, grid, dim3(32, GT::WARPS), GT::SMEM, st, tmX, tmU,
                              tmA, a);
}
}  // namespace

// About the time of an RK4 step by pairs over that by the four stage kernels, which
// store their own ghost values: 0.68 for each point that the tiles' 28 x 8 columns
// span over those of the grid, 0.2 where every tile lies at an r end (its warps take
// the general path), and a start that shows below some tens of tile planes per SM.
// Fitted to 47 grids, 22 x 65 x 513 to 2048 x 129 x 257.  us per step, pairs / stages
// (tile planes per SM): 128 x 33 x 65 (9) 119 / 100, 64 x 65 x 129 (21) 230 / 197, 256 x
// 33 x 65 (17) 177 / 181, 512 x 33 x 65 (33) 296 / 302, 301 x 46 x 90 (40) 334 / 377,
// 64 x 129 x 257 (83) 711 / 674, 384 x 65 x 129 (97) 691 / 866, 1024 x 65 x 129 (256)
// 1853 / 2149, 2048 x 129 x 257 (2048) 13064 / 17173.  On the wrong side of the line by
// 1 to 8 %: 160 x 33 x 65, 320 x 33 x 65, 80 x 65 x 129, 1000 x 17 x 33.
static double pair_time(const Grid& g) {
  const int cols = g.NI - 2, rows = g.NJ - 6;
  const int tx = (cols + PO - 1) / PO, ty = (rows + TJ - 1) / TJ;
  const double tiles = (double)tx * ty;
  const double padding = tiles * (PO * TJ) / ((double)cols * rows), ends = tx > 2 ? 2.0 / tx : 1.0;
  return 0.68 * padding + 3.5 * 148 / (tiles * (g.Nz - 1)) + 0.2 * ends;
}
bool rk4_pairs_pay(const Grid& g) { return pair_time(g) < 1.0; }
// a step whose result has to be copied back from the second u buffer: us, pairs and
// copy / stages: 512 x 33 x 65 338 / 301, 192 x 65 x 129 470 / 461, 576 x 33 x 65 362 / 405,
// 384 x 65 x 129 793 / 855, 2048 x 129 x 257 14788 / 17160
bool rk4_pairs_and_copy_pay(const Grid& g) { return pair_time(g) < 0.815; }

int launch_rk4_pair(int pair, const PairLaunch& L, const double* rsg, int* err, cudaStream_t st) {
  if (pair == 0)
    return L.metric_kind == MK_KS ? pair_launch<0, MK_KS>(L, rsg, err, st) : pair_launch<0, MK_SCHW>(L, rsg, err, st);
  return L.metric_kind == MK_KS ? pair_launch<1, MK_KS>(L, rsg, err, st) : pair_launch<1, MK_SCHW>(L, rsg, err, st);
}

}  // namespace kg
