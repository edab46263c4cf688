// eig.cuh — small dense Hermitian eigensolvers for device code: one matrix per
// thread (2 to 5 bands), or one matrix per group of N lanes (8 and 16 bands).
#pragma once
#include "dev.cuh"

namespace edus {

// Hermitian eigenvectors by cyclic Jacobi; Z columns are eigenvectors,
// eigenvalues ascending (Armadillo eig_sym in Observables_MPI.h:294).
template <int N>
__device__ void eig_herm_dev(double2* A, double2* Z) {
  for (int i = 0; i < N; i++)
    for (int j = 0; j < N; j++) Z[i * N + j] = (i == j) ? cmk(1., 0.) : cz();
  for (int sweep = 0; sweep < 50; sweep++) {
    double off = 0, diag = 0;
    for (int i = 0; i < N; i++) {
      diag += A[i * N + i].x * A[i * N + i].x;
      for (int j = i + 1; j < N; j++) off += A[i * N + j].x * A[i * N + j].x + A[i * N + j].y * A[i * N + j].y;
    }
    if (off <= 1e-34 * (diag + 1e-300)) break;
    for (int p = 0; p < N; p++)
      for (int q = p + 1; q < N; q++) {
        double2 apq = A[p * N + q];
        double mag = hypot(apq.x, apq.y);
        if (mag < 1e-300) continue;
        double app = A[p * N + p].x, aqq = A[q * N + q].x;
        double2 ph = cmk(apq.x / mag, apq.y / mag);
        double theta = 0.5 * atan2(2.0 * mag, aqq - app);
        double s, c;
        sincos(theta, &s, &c);
        double2 sp = cscale(ph, s), sc = cscale(cconj(ph), s);
        for (int k = 0; k < N; k++) {
          double2 akp = A[k * N + p], akq = A[k * N + q];
          A[k * N + p] = csub(cscale(akp, c), cmul(sc, akq));
          A[k * N + q] = cadd(cmul(sp, akp), cscale(akq, c));
        }
        for (int k = 0; k < N; k++) {
          double2 apk = A[p * N + k], aqk = A[q * N + k];
          A[p * N + k] = csub(cscale(apk, c), cmul(sp, aqk));
          A[q * N + k] = cadd(cmul(sc, apk), cscale(aqk, c));
        }
        A[p * N + q] = cz();
        A[q * N + p] = cz();
        A[p * N + p].y = 0;
        A[q * N + q].y = 0;
        for (int k = 0; k < N; k++) {
          double2 zkp = Z[k * N + p], zkq = Z[k * N + q];
          Z[k * N + p] = csub(cscale(zkp, c), cmul(sc, zkq));
          Z[k * N + q] = cadd(cmul(sp, zkp), cscale(zkq, c));
        }
      }
  }
  for (int i = 1; i < N; i++) {
    int j = i;
    while (j > 0 && A[(j - 1) * N + (j - 1)].x > A[j * N + j].x) {
      double2 t = A[(j - 1) * N + (j - 1)];
      A[(j - 1) * N + (j - 1)] = A[j * N + j];
      A[j * N + j] = t;
      for (int r = 0; r < N; r++) {
        double2 z = Z[r * N + j - 1];
        Z[r * N + j - 1] = Z[r * N + j];
        Z[r * N + j] = z;
      }
      j--;
    }
  }
}

// The same cyclic Jacobi with N lanes of a warp per matrix (N = 8 or 16; 32 / N
// matrices per warp): the rotations follow one another in the same order and
// every entry is updated by the same expression, so the eigenvectors are those
// of eig_herm_dev. A thread per matrix is a chain of 120 rotations a sweep
// with 16-band rows in local memory; here lane r updates row r (then column r)
// of the matrix in shared memory.
//
// A, Z: this group's matrices [N][N + 1] in shared memory (the odd row stride in
// 16-byte words spreads a column over the banks), A filled and visible to the
// warp. r: lane within the group. All 32 lanes of the warp call it together;
// groups whose matrix has converged keep stepping without writing.
template <int N>
struct EigGroup {
  static constexpr int LD = N + 1;
  static constexpr int WORDS = 2 * N * LD;  // double2 of A and Z
};

// Ascending order: the insertion sort of the diagonal, its column swaps on each
// lane's row of Z.
template <int N>
__device__ __forceinline__ void eig_sort_group(const double2* A, double2* Z, int r) {
  constexpr int LD = EigGroup<N>::LD;
  __syncwarp();
  double ev[N];
#pragma unroll
  for (int i = 0; i < N; i++) ev[i] = A[i * LD + i].x;
#pragma unroll
  for (int i = 1; i < N; i++) {
#pragma unroll
    for (int j = i; j > 0; j--) {
      if (!(ev[j - 1] > ev[j])) break;
      const double t = ev[j - 1];
      ev[j - 1] = ev[j];
      ev[j] = t;
      const double2 z = Z[r * LD + j - 1];
      Z[r * LD + j - 1] = Z[r * LD + j];
      Z[r * LD + j] = z;
    }
  }
  __syncwarp();
}

template <int N>
__device__ void eig_herm_group(double2* A, double2* Z, int r) {
  constexpr int LD = EigGroup<N>::LD;
  for (int j = 0; j < N; j++) Z[r * LD + j] = (r == j) ? cmk(1., 0.) : cz();
  bool live = true;
  for (int sweep = 0; sweep < 50; sweep++) {
    double off = 0, diag = 0;
    for (int i = 0; i < N; i++) {
      diag += A[i * LD + i].x * A[i * LD + i].x;
      for (int j = i + 1; j < N; j++) off += A[i * LD + j].x * A[i * LD + j].x + A[i * LD + j].y * A[i * LD + j].y;
    }
    if (off <= 1e-34 * (diag + 1e-300)) live = false;
    if (!__any_sync(0xffffffffu, live)) break;
    for (int p = 0; p < N; p++)
      for (int q = p + 1; q < N; q++) {
        const double2 apq = A[p * LD + q];
        const double mag = hypot(apq.x, apq.y);
        const bool on = live && !(mag < 1e-300);  // uniform over the group
        const double app = A[p * LD + p].x, aqq = A[q * LD + q].x;
        const double2 ph = cmk(apq.x / mag, apq.y / mag);
        const double theta = 0.5 * atan2(2.0 * mag, aqq - app);
        double s, c;
        sincos(theta, &s, &c);
        const double2 sp = cscale(ph, s), sc = cscale(cconj(ph), s);
        __syncwarp();
        if (on) {
          const double2 akp = A[r * LD + p], akq = A[r * LD + q];
          A[r * LD + p] = csub(cscale(akp, c), cmul(sc, akq));
          A[r * LD + q] = cadd(cmul(sp, akp), cscale(akq, c));
          const double2 zkp = Z[r * LD + p], zkq = Z[r * LD + q];
          Z[r * LD + p] = csub(cscale(zkp, c), cmul(sc, zkq));
          Z[r * LD + q] = cadd(cmul(sp, zkp), cscale(zkq, c));
        }
        __syncwarp();
        if (on) {
          const double2 apk = A[p * LD + r], aqk = A[q * LD + r];
          double2 np = csub(cscale(apk, c), cmul(sp, aqk));
          double2 nq = cadd(cmul(sc, apk), cscale(aqk, c));
          // the pivot pair is zero and the diagonal real
          if (r == q) np = cz();
          if (r == p) nq = cz();
          if (r == p) np.y = 0;
          if (r == q) nq.y = 0;
          A[p * LD + r] = np;
          A[q * LD + r] = nq;
        }
        __syncwarp();
      }
  }
  eig_sort_group<N>(A, Z, r);
}

// The same rotations with the disjoint ones side by side, again N lanes per matrix.
// The cyclic order (0,1), (0,2), .. (1,2), .. only needs a rotation to follow those
// that share an index with it, and these have a smaller p + q: the pairs of one
// p + q are disjoint and may be taken together, 2 N - 3 steps a sweep (13 and 29)
// in place of N (N - 1) / 2 (28 and 120) and the same eigenvectors but for the
// rounding. Lane m forms the rotation of pair m; then every lane applies all of
// them to its row and, after a warp barrier, to its column. With d = aqq - app
// and h = sqrt(d^2 + 4 |apq|^2) the angle atan2(2 |apq|, d) / 2 of eig_herm_group has
// max(c, s)^2 = (h + |d|) / 2h and c s = |apq| / h: two reciprocal roots one after
// the other instead of hypot, atan2 and sincos, and one correction of
// c^2 + |s|^2 to 1. Bound by the chain of steps and, with 16 bands, by shared
// memory. 4096 8-band matrices: 80.5 us, 168 with eig_herm_group. Observables of the
// velocity gauge only: the Coulomb mean field's n_cond > 1e-20 switch and the FP32
// stages of a mixed batch, whose ground state comes from these eigenvectors, carry
// a changed last bit to 1e-9 and more.
template <int N>
__device__ void eig_herm_wave(double2* A, double2* Z, int r) {
  constexpr int LD = EigGroup<N>::LD, P = N / 2;
  for (int j = 0; j < N; j++) Z[r * LD + j] = (r == j) ? cmk(1., 0.) : cz();
  bool live = true;
  for (int sweep = 0; sweep < 50; sweep++) {
    double off = 0., diag = A[r * LD + r].x * A[r * LD + r].x;
#pragma unroll
    for (int j = 1; j < N; j++)
      if (j > r) off += A[r * LD + j].x * A[r * LD + j].x + A[r * LD + j].y * A[r * LD + j].y;
#pragma unroll
    for (int o = N / 2; o > 0; o /= 2) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      diag += __shfl_xor_sync(0xffffffffu, diag, o);
    }
    // (a converged matrix goes on with identities until the others of its warp are)
    live = live && !(off <= 1e-34 * (diag + 1e-300));
    if (!__any_sync(0xffffffffu, live)) break;
#pragma unroll 1
    for (int t = 1; t <= 2 * N - 3; t++) {  // p + q
      const int p0 = t < N ? 0 : t - N + 1, cnt = (t + 1) / 2 - p0;
      double c = 1., sx = 0., sy = 0.;  // cos, and sin times the phase of apq
      if (r < cnt) {
        const int p = p0 + r, q = t - p;
        const double2 apq = A[p * LD + q];
        const double d = A[q * LD + q].x - A[p * LD + p].x;
        const double m2 = apq.x * apq.x + apq.y * apq.y;
        if (live && m2 > 1e-290) {
          const double rh = rsqrt(d * d + 4. * m2);     // 1 / h
          const double x = 0.5 + 0.5 * fabs(d) * rh;    // the larger of c^2, s^2
          const double rb = rsqrt(x), rm = rsqrt(m2);
          const double big = x * rb, small = m2 * rm * rh * rb;
          const double f = d >= 0. ? rh * rb : big * rm;  // s / |apq|
          c = d >= 0. ? big : small;
          sx = apq.x * f;
          sy = apq.y * f;
          const double n1 = 1. + 0.5 * fma(-sy, sy, fma(-sx, sx, fma(-c, c, 1.)));
          c *= n1;
          sx *= n1;
          sy *= n1;
        }
      }
      __syncwarp();
      double pc[P], px[P], py[P];
#pragma unroll
      for (int m = 0; m < P; m++)
        if (m < cnt) {
          pc[m] = __shfl_sync(0xffffffffu, c, m, N);
          px[m] = __shfl_sync(0xffffffffu, sx, m, N);
          py[m] = __shfl_sync(0xffffffffu, sy, m, N);
          const int p = p0 + m, q = t - p;
          const double2 sp = cmk(px[m], py[m]), sc = cmk(px[m], -py[m]);
          const double2 akp = A[r * LD + p], akq = A[r * LD + q];
          A[r * LD + p] = csub(cscale(akp, pc[m]), cmul(sc, akq));
          A[r * LD + q] = cadd(cmul(sp, akp), cscale(akq, pc[m]));
          const double2 zkp = Z[r * LD + p], zkq = Z[r * LD + q];
          Z[r * LD + p] = csub(cscale(zkp, pc[m]), cmul(sc, zkq));
          Z[r * LD + q] = cadd(cmul(sp, zkp), cscale(zkq, pc[m]));
        }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < P; m++)
        if (m < cnt) {
          const int p = p0 + m, q = t - p;
          const double2 sp = cmk(px[m], py[m]), sc = cmk(px[m], -py[m]);
          const double2 apk = A[p * LD + r], aqk = A[q * LD + r];
          double2 np = csub(cscale(apk, pc[m]), cmul(sp, aqk));
          double2 nq = cadd(cmul(sc, apk), cscale(aqk, pc[m]));
          // the pivot pair is zero and the diagonal real
          if (r == q) np = cz();
          if (r == p) nq = cz();
          if (r == p) np.y = 0;
          if (r == q) nq.y = 0;
          A[p * LD + r] = np;
          A[q * LD + r] = nq;
        }
      __syncwarp();
    }
  }
  eig_sort_group<N>(A, Z, r);
}

}  // namespace edus
