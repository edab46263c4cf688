// obs.cuh — the fields an output instant sums over k, and the record made of them.
#pragma once
#include "dev.cuh"
#include "kernels.hpp"

namespace edus {

// fields of a partial: populations, then per component x J1 re, J1 im, J2 im,
// TA re, TA im, polarisation re, im, then max and min
constexpr int kFX = kMaxBands;
constexpr int kPerX = 7;
constexpr int kFMax = kFX + 3 * kPerX, kFMin = kFMax + 1;
constexpr int kFields = kFMin + 1;

__device__ __forceinline__ double obs_op(int f, double a, double b) {
  return f == kFMax ? fmax(a, b) : (f == kFMin ? fmin(a, b) : a + b);
}

// One warp: value f of 128 consecutive entries (four per lane) as a binary tree
// over 128; the result is lane 0's.
__device__ __forceinline__ double tree128(int f, double v0, double v1, double v2, double v3) {
  double x = obs_op(f, obs_op(f, v0, v2), obs_op(f, v1, v3));
  for (int s = 16; s > 0; s >>= 1) x = obs_op(f, x, __shfl_down_sync(0xffffffffu, x, s));
  return x;
}

// Field v of a block that carries N populations, in the partial's numbering.
template <int N>
__device__ __forceinline__ int field_no(int v) { return v < N ? v : kFX + (v - N); }

// The record's sums from the totals T(f) of every field; returns n_cond.
template <class F>
__device__ __forceinline__ double obs_fill(ObsRecord& rec, const F& T, int n, int nk, int nbands, double scaleJ, double scaleTA) {
  const double inv = 1. / nk;
  double trace = -(double)nbands;
  double nc = 0;
  for (int i = 0; i < n; i++) {
    double v = T(i) * inv;
    trace += v;
    if (i < nbands) v = 1.0 - v;
    rec.pop[i] = v;
    if (v > nc) nc = v;
  }
#pragma unroll
  for (int x = 0; x < 3; x++) {
    const int f = kFX + kPerX * x;
    rec.J1[2 * x] = T(f) * scaleJ;
    rec.J1[2 * x + 1] = T(f + 1) * scaleJ;
    rec.J2[x] = -2. * (T(f + 2) * scaleJ);
    rec.tabs[2 * x] = T(f + 3) * scaleTA * inv;
    rec.tabs[2 * x + 1] = T(f + 4) * scaleTA * inv;
    rec.pol[2 * x] = T(f + 5) * inv;
    rec.pol[2 * x + 1] = T(f + 6) * inv;
  }
  rec.trace_dev = trace;
  rec.p_cond_max = T(kFMax);
  rec.p_min = T(kFMin);
  rec.n_cond = nc;
  return nc;
}

}  // namespace edus
