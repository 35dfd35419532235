// kg_chunk.h -- phi planes per chunk of the kernels that march through planes (host
// code, no CUDA).
#pragma once

namespace kg {

// The chunk length of `planes` planes, at most `longest`, with the least cost(c, m),
// c planes in each of m chunks; the longest one among equals.  The lengths tried are
// those of equal chunks, ceil(planes / n) for each number n of chunks, and at most
// `longest` of them differ, so the time does not grow with the planes (it is paid at
// every launch; with one try per n it was 5 us at 1024 planes and 330 us at 70000).
template <class F>
inline int best_chunk(int planes, int longest, F cost) {
  int best = planes;
  double least = 1e300;
  for (int most = longest < planes ? longest : planes; most >= 1;) {
    const int n = (planes + most - 1) / most, c = (planes + n - 1) / n;
    const double t = cost(c, (planes + c - 1) / c);
    if (t < least) {
      least = t;
      best = c;
    }
    most = c - 1;
  }
  return best;
}

// Phi planes per chunk of a marching kernel: `planes` planes of each of `tiles`
// (r, theta) tiles, on `slots` CTAs that run at once, at most `longest` planes.
// A chunk of c planes costs c + 1 plane times (its two halo planes and its
// prologue overlap the other CTA of the SM) and the launch's last wave a quarter
// of a chunk, so the rule takes the c that minimises
//   max(1, tiles * chunks / slots + 1/4) * (c + 1);
// a grid whose tiles alone leave SMs idle gets short chunks, a large one the
// longest.  Constants fitted to a sweep of 19 lengths over ten grids from
// 64 x 17 x 33 to 1024 x 65 x 129 (within 2 % of the best length on average, 14 %
// at worst).  Event-timed us per launch with about 32 planes a chunk on every grid
// (64 in the fused PIRK stage 1) and every stored row computed, and now, with these
// chunks and the interior rows alone: 64 x 17 x 33 PIRK2 stage 2 53.7 / 11.2 and fused
// stage 1 98.4 / 19.1, 256 x 33 x 65 78.4 / 37.2 and 103.0 / 47.4, RK4 stage 2 106 / 55.4.
inline int phi_chunk(int planes, long long tiles, int slots, int longest) {
  return best_chunk(planes, longest, [&](int c, int m) {
    const double waves = (double)tiles * m / slots + 0.25;
    return (waves > 1.0 ? waves : 1.0) * (c + 1);
  });
}

// The same for the RK4 pairs (kg_pair.cu).  One CTA runs on an SM at a time, so its
// start shows: a chunk costs c + 3 plane times, a launch whole waves of them, and
// half a chunk at the end behind the tiles at the r ends, whose warps take the
// general path.  At most 24 planes: longer chunks measured slower on large grids
// (1024 x 65 x 129, pair 0: 661 us at 24, 699 at 32, 712 at 43, 709 at 16).
inline int pair_chunk(int planes, long long tiles) {
  return best_chunk(planes, 24, [&](int c, int m) { return ((double)((tiles * m + 147) / 148) + 0.5) * (c + 3); });
}

}  // namespace kg
