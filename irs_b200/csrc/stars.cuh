// Star-field generation on the device.
//
// Same draw protocol as the reference (include/star.cuh:40-107): star i owns
// the curand XORWOW sequence (seed, subsequence i, offset 0); a rectangular
// field takes two uniform doubles for x1 and x2 in [-corner, corner]; a
// circular field takes an angle U*2pi and a radius sqrt(U)*|corner|; the mass
// is then drawn from the mass function with one more uniform double. The curand
// state lives in registers only (the reference keeps one state per star in
// global memory; the draws are the same).
#pragma once
#include "common.cuh"
#include "massfn.cuh"
#include "params.hpp"

#include <curand_kernel.h>

namespace irsb {

// What star i of a field is drawn with.
template <typename T>
struct StarDraw {
  int seed, rectangular, mf_kind;
  cplx<T> corner;
  T m_lower, m_upper, m_solar;
};

template <typename T>
__device__ __forceinline__ StarRec<T> draw_star(const StarDraw<T>& d, int i) {
  curandState st;
  curand_init((unsigned long long)d.seed, (unsigned long long)i, 0ULL, &st);
  T x1, x2;
  if (d.rectangular) {
    x1 = T(curand_uniform_double(&st) * 2 * d.corner.re - d.corner.re);
    x2 = T(curand_uniform_double(&st) * 2 * d.corner.im - d.corner.im);
  } else {
    T a = T(curand_uniform_double(&st) * 2 * kPi<T>);
    T r = T(sqrt(curand_uniform_double(&st)) * cabs_(d.corner));
    x1 = r * xcos(a);
    x2 = r * xsin(a);
  }
  T p = T(curand_uniform_double(&st));
  StarRec<T> s;
  s.x = x1;
  s.y = x2;
  s.m = mf_mass<T>(d.mf_kind, p, d.m_lower, d.m_upper, d.m_solar);
  return s;
}

template <typename T>
__global__ void __launch_bounds__(256) generate_stars_kernel(StarRec<T>* __restrict__ stars, int n, StarDraw<T> d) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) stars[i] = draw_star(d, i);
}

// The fields of R realizations in one launch: realization r owns the stars
// [off[r], off[r + 1]). Bound by curand_init's skip-ahead, a long dependent
// chain per star that one field of 8e4 stars leaves mostly exposed: a launch
// per field took 5.5 ms for 24 fields of 1.9e6 stars in all (B200), this one
// 3.4 ms.
template <typename T>
__global__ void __launch_bounds__(256) generate_stars_batch(StarRec<T>* __restrict__ stars, int R,
                                                            const long long* __restrict__ off,
                                                            const StarDraw<T>* __restrict__ draw) {
  const long long n = off[R];
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = R - 1;  // last realization with off[r] <= q
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    stars[q] = draw_star(draw[lo], int(q - off[lo]));
  }
}

}  // namespace irsb
