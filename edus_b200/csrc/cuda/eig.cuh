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
  // ascending order: the insertion sort of the diagonal, its column swaps on
  // each lane's row of Z
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

}  // namespace edus
