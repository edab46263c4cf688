// layout.cu — the reference's [k][i][j](component) layout against the device's
// upper-triangle planes [component][e][k].
//
// Both kernels are one pass over the larger side, bound by that traffic: a block
// takes 32 k points, so plane accesses are runs of 32 entries and the other
// side is one contiguous piece of 32 matrices. The host did the same a matrix at
// a time with strided accesses (2.7 ms for the tables of a 96 x 96 8-band state,
// 5 ms for those of a 144 x 144 2-band model; 10 and 20 us here).
#include "kernels.hpp"

namespace edus {
namespace {

constexpr int kLayoutK = 32, kLayoutThreads = 256;

// planes[x][e][k] = src[k][i][j][x], i <= j (full: every (i, j), e = i n + j)
template <class T>
__global__ void __launch_bounds__(kLayoutThreads) k_to_planes(const double2* __restrict__ src, int nk, int n, int comps, int full,
                                                              T* __restrict__ dst) {
  const int k0 = blockIdx.x * kLayoutK, ne = full ? n * n : n * (n + 1) / 2;
  for (int t = threadIdx.x; t < kLayoutK * ne * comps; t += kLayoutThreads) {
    const int k = k0 + t % kLayoutK, p = t / kLayoutK, x = p / ne, e = p - x * ne;
    if (k >= nk) continue;
    int i = 0, j = 0;
    if (full) {
      i = e / n;
      j = e - i * n;
    } else {
      int r = e;
      while (r >= n - i) {
        r -= n - i;
        i++;
      }
      j = i + r;
    }
    const double2 v = src[(((size_t)k * n + i) * n + j) * comps + x];
    T o;
    o.x = v.x;
    o.y = v.y;
    dst[(size_t)p * nk + k] = o;
  }
}

// dst[k][i][j] = P_e (+ Q_e), the lower entry conjugated
__global__ void __launch_bounds__(kLayoutThreads) k_from_planes(const double2* __restrict__ P, const double2* __restrict__ Q, int nk,
                                                                int n, double2* __restrict__ dst) {
  const int k0 = blockIdx.x * kLayoutK, kn = min(kLayoutK, nk - k0);
  for (int t = threadIdx.x; t < kn * n * n; t += kLayoutThreads) {
    const int m = t / (n * n), ij = t - m * n * n, i = ij / n, j = ij - i * n;
    const int lo = i < j ? i : j, hi = i < j ? j : i;
    const size_t o = (size_t)tri_index(lo, hi, n) * nk + k0 + m;
    double2 v = P[o];
    if (Q) v = cadd(v, Q[o]);
    dst[(size_t)k0 * n * n + t] = i > j ? cconj(v) : v;
  }
}

}  // namespace

cudaError_t launch_to_planes(const double2* src, int nk, int n, int comps, bool full, double2* dst, cudaStream_t s) {
  k_to_planes<double2><<<(nk + kLayoutK - 1) / kLayoutK, kLayoutThreads, 0, s>>>(src, nk, n, comps, full, dst);
  return cudaGetLastError();
}
cudaError_t launch_to_planes(const double2* src, int nk, int n, int comps, bool full, float2* dst, cudaStream_t s) {
  k_to_planes<float2><<<(nk + kLayoutK - 1) / kLayoutK, kLayoutThreads, 0, s>>>(src, nk, n, comps, full, dst);
  return cudaGetLastError();
}
cudaError_t launch_from_planes(const double2* P, const double2* Q, int nk, int n, double2* dst, cudaStream_t s) {
  k_from_planes<<<(nk + kLayoutK - 1) / kLayoutK, kLayoutThreads, 0, s>>>(P, Q, nk, n, dst);
  return cudaGetLastError();
}

}  // namespace edus
