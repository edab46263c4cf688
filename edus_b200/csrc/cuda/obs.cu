// obs.cu — observables of a single solve at an output instant (FP64, sm_100a):
// populations (headers/Observables_MPI.h:217-484), J1 / J2 (:668-775), the
// transient absorption (:559-598) and the polarisation, summed over k.
//
//   k_obs<N>     1 to 5 bands: one thread per k point.
//   k_obs_el<N>  8 and 16 bands: one thread per (k point, full-matrix entry).
//                A thread per k point needs N^3 products one after the other
//                on rows in local memory (measured 2.6 ms an instant for 16 bands
//                on 30 x 34, 0.2 ms for 8 bands on 96 x 96; 48 and 53 us
//                in this form).
//   k_eig_rows   with a renormalised H and 8 or 16 bands: its eigenvectors, N lanes
//                per k point (eig.cuh), into a scratch that k_obs_el reads.
//
// Every block writes the partial sums of its k points; the last block to finish
// adds them in a fixed order and writes the output record: no second launch, no
// host round trip.
#include "dev.cuh"
#include "dyn.cuh"
#include "eig.cuh"
#include "kernels.hpp"
#include "obs.cuh"

namespace edus {

namespace {

template <int N>
struct Tri {
  static constexpr int NT = N * (N + 1) / 2;
  static __device__ __forceinline__ int idx(int i, int j) { return i * N - (i * (i - 1)) / 2 + (j - i); }
};

// Sums of one k point, thread or block in k_obs.
struct ObsPart {
  double pop[kMaxBands];
  double2 J1[3], J2[3], TA[3], PL[3];
  double pmax, pmin;
};

__device__ __forceinline__ void obs_zero(ObsPart& p) {
  for (int i = 0; i < kMaxBands; i++) p.pop[i] = 0;
  for (int x = 0; x < 3; x++) p.J1[x] = p.J2[x] = p.TA[x] = p.PL[x] = cz();
  p.pmax = 0;
  p.pmin = 1.0;
}
__device__ __forceinline__ void obs_add(ObsPart& d, const ObsPart& o, int n) {
  for (int i = 0; i < n; i++) d.pop[i] += o.pop[i];
  for (int x = 0; x < 3; x++) {
    d.J1[x] = cadd(d.J1[x], o.J1[x]);
    d.J2[x] = cadd(d.J2[x], o.J2[x]);
    d.TA[x] = cadd(d.TA[x], o.TA[x]);
    d.PL[x] = cadd(d.PL[x], o.PL[x]);
  }
  d.pmax = fmax(d.pmax, o.pmax);
  d.pmin = fmin(d.pmin, o.pmin);
}

struct ObsArgs {
  const double2* rho;
  const double2* hr;
  const double2* uev;  // eigenvector rows of hr (k_obs_el), else null
  int want_current, want_tabs;
  double* part;        // ObsPart per block (k_obs), or [kFields][gridDim.x] (k_obs_el)
  unsigned int* done;
  double scaleJ, scaleTA;
  ObsRecord rec;
  ObsRecord* log;
  double* ncond_dev;
  double* pcmax_dev;
  int per;             // k_obs_el: sub-tiles per block
  // adaptive step on the device: the instant is taken only when dyn->obs_now,
  // with the clock, field and step of *dyn, into record dyn->nlog of log
  const DynStep* dyn;
};

constexpr int kObsThreads = 128;
static_assert(kFields * sizeof(double) <= sizeof(ObsPart), "partials are sized by the larger form");
// blocks of k_obs_el: enough for three 256- or two 512-thread blocks on every SM
constexpr int kObsElBlocks = 512;

// The output record from the totals T(f) of every field (one thread).
template <int N, class F>
__device__ __forceinline__ void obs_record(const DevTables& tb, const ObsArgs& a, const F& T) {
  ObsRecord rec = a.rec;
  ObsRecord* slot = a.log;
  if (a.dyn) {
    const DynStep* d = a.dyn;
    rec.t = d->t;
    rec.dt = d->dt;
    for (int x = 0; x < 3; x++) {
      rec.EF_pump[x] = d->EF_last[0][x];
      rec.EF_probe[x] = d->EF_last[1][x];
    }
    slot = (a.log && d->nlog < d->log_cap) ? a.log + d->nlog : nullptr;
  }
  const double nc = obs_fill(rec, T, N, tb.nk, tb.nbands, a.scaleJ, a.scaleTA);
  if (slot) *slot = rec;
  if (a.ncond_dev) *a.ncond_dev = nc;
  if (a.pcmax_dev) *a.pcmax_dev = T(kFMax);
  *a.done = 0u;
}

// The block's partial is written; the last block sums all of them and writes
// the record. T: kFields doubles of shared memory.
template <int N>
__device__ __forceinline__ void obs_finish(const DevTables& tb, const ObsArgs& a, double* T) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int lane = threadIdx.x % 32, nw = blockDim.x / 32;
  const int np = gridDim.x;
  for (int v = threadIdx.x / 32; v < N + 3 * kPerX + 2; v += nw) {
    const int f = field_no<N>(v);
    const double* row = a.part + (size_t)f * np;
    const double id = f == kFMin ? 1.0 : 0.0;
    double t[4] = {id, id, id, id};
    for (int b = lane; b < np; b += 128)
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (b + 32 * j < np) t[j] = obs_op(f, t[j], __ldcg(row + b + 32 * j));
    const double x = tree128(f, t[0], t[1], t[2], t[3]);
    if (lane == 0) T[f] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) obs_record<N>(tb, a, [&](int f) { return T[f]; });
}

// One thread per k point.
template <int N>
__global__ void __launch_bounds__(kObsThreads) k_obs(DevTables tb, const DevConsts* __restrict__ cst, ObsArgs a) {
  constexpr int NT = Tri<N>::NT;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int nk = tb.nk;
  __shared__ ObsPart sp[kObsThreads];
  __shared__ bool last;
  ObsPart my;
  obs_zero(my);
  const double2* rho = a.rho;
  ObsPart* part = reinterpret_cast<ObsPart*>(a.part);
  const double2* hr = a.hr;
  pdl_wait();
  if (a.dyn && !a.dyn->obs_now) return;  // uniform: no instant at this step
  if (k < nk) {
    double2 P[NT];
#pragma unroll
    for (int e = 0; e < NT; e++) P[e] = rho[(size_t)e * nk + k];
    auto Pf = [&](int i, int j) -> double2 { return (i <= j) ? P[Tri<N>::idx(i, j)] : cconj(P[Tri<N>::idx(j, i)]); };
    double2 Ue[N * N];
    if (hr) {
      double2 A[N * N], Z[N * N];
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
          const double2 v = hr[(size_t)Tri<N>::idx(i, j) * nk + k];
          A[i * N + j] = v;
          A[j * N + i] = cconj(v);
        }
      eig_herm_dev<N>(A, Z);
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) Ue[i * N + j] = cconj(Z[j * N + i]);
    } else {
#pragma unroll
      for (int e = 0; e < N * N; e++) Ue[e] = tb.U[(size_t)e * nk + k];
    }
#pragma unroll
    for (int c = 0; c < N; c++) {
      double2 acc = cz();
#pragma unroll
      for (int ii = 0; ii < N; ii++) {
        double2 m = cz();
#pragma unroll
        for (int jj = 0; jj < N; jj++) m = cadd(m, cmul(Pf(ii, jj), Ue[c * N + jj]));
        acc = cadd(acc, cmul(cconj(Ue[c * N + ii]), m));
      }
      const double Pik = acc.x;
      my.pop[c] = Pik;
      if (c < tb.nbands) {
        my.pmax = fmax(my.pmax, fabs(1. - Pik));
        my.pmin = fmin(my.pmin, 1. - Pik);
      } else {
        my.pmax = fmax(my.pmax, fabs(Pik));
        my.pmin = fmin(my.pmin, Pik);
      }
    }
    if (a.want_current) {
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
          const int e = Tri<N>::idx(i, j);
          double2 ge[3];
          if (hr) {
            ge[0] = ge[1] = ge[2] = cz();
            const double2 h0 = hr[(size_t)e * nk + k];
            for (int b = 0; b < tb.nnb; b++) {
              const int kb = tb.nbr[(size_t)b * nk + k];
              const double2 d = csub(hr[(size_t)e * nk + kb], h0);
#pragma unroll
              for (int x = 0; x < 3; x++) ge[x] = cadd(ge[x], cscale(d, cst->wb[b] * cst->bvec[b][x]));
            }
          } else {
#pragma unroll
            for (int x = 0; x < 3; x++) ge[x] = tb.GE[(size_t)(x * NT + e) * nk + k];
          }
#pragma unroll
          for (int x = 0; x < 3; x++) {
            my.J1[x] = cadd(my.J1[x], cmul(P[e], ge[x]));
            if (i != j) my.J1[x] = cadd(my.J1[x], cmul(cconj(P[e]), cconj(ge[x])));
          }
        }
      const double2* Hs = hr ? hr : tb.H;
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
          const double2 pij = Pf(i, j);
#pragma unroll
          for (int l = 0; l < N; l++) {
            const double2 hil = (i <= l) ? Hs[(size_t)Tri<N>::idx(i, l) * nk + k] : cconj(Hs[(size_t)Tri<N>::idx(l, i) * nk + k]);
            const double2 ph = cmul(pij, hil);
            const int lo = j < l ? j : l, hi = j < l ? l : j;
            // D_jl: the stored upper entry, conjugated below the diagonal for Hermitian dipoles
            const bool cj = tb.herm_dip && j > l;
#pragma unroll
            for (int x = 0; x < 3; x++) {
              const double2 ds = tb.D[(size_t)(x * NT + Tri<N>::idx(lo, hi)) * nk + k];
              const double2 d = cj ? cconj(ds) : ds;
              my.J2[x] = cadd(my.J2[x], cmulc(ph, d));
            }
          }
        }
    }
    // polarisation: Tr(D_x rho) = sum_ij D_x,ij P_ij in the reference's P[k][i][j] = rho_ji
    // convention (lower D entries: D_ji = D_ij, or conj(D_ij) for Hermitian dipoles)
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) {
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        const bool cj = tb.herm_dip && i > j;
        const double2 pij = Pf(i, j);
#pragma unroll
        for (int x = 0; x < 3; x++) {
          const double2 ds = tb.D[(size_t)(x * NT + Tri<N>::idx(lo, hi)) * nk + k];
          my.PL[x] = cadd(my.PL[x], cmul(cj ? cconj(ds) : ds, pij));
        }
      }
    if (a.want_tabs)
      for (int i = 0; i < tb.nch; i++)
        for (int j = tb.nch; j < N; j++) {
          const int e = Tri<N>::idx(i, j);
          for (int x = 0; x < 3; x++)
            my.TA[x] = csub(my.TA[x], cmul(cscale(tb.D[(size_t)(x * NT + e) * nk + k], 2.), P[e]));
        }
  }
  sp[threadIdx.x] = my;
  __syncthreads();
  for (int s = kObsThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) obs_add(sp[threadIdx.x], sp[threadIdx.x + s], N);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[blockIdx.x] = sp[0];
    __threadfence();
    const unsigned int prev = atomicAdd(a.done, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  // last block: fixed-order reduction of all block partials
  __threadfence();
  ObsPart t;
  obs_zero(t);
  for (int b = threadIdx.x; b < gridDim.x; b += kObsThreads) obs_add(t, part[b], N);
  sp[threadIdx.x] = t;
  __syncthreads();
  for (int s = kObsThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) obs_add(sp[threadIdx.x], sp[threadIdx.x + s], N);
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  const ObsPart& S = sp[0];
  obs_record<N>(tb, a, [&](int f) {  // (f is a constant at every use)
    if (f < kFX) return S.pop[f];
    if (f >= kFMax) return f == kFMax ? S.pmax : S.pmin;
    const int x = (f - kFX) / kPerX, m = (f - kFX) % kPerX;
    const double2 z = m < 2 ? S.J1[x] : (m < 3 ? S.J2[x] : (m < 5 ? S.TA[x] : S.PL[x]));
    return m == 0 || m == 3 || m == 5 ? z.x : z.y;
  });
}

// One thread per (k point, entry (b, l) of the full matrices), KO k points at a
// time; a block takes a run of a.per such sub-tiles. J2_x = sum_bl conj(D^x_bl)
// Q_bl with Q = P^T H formed once for the three components; the population of
// band b is the sum over l of its terms conj(U_bl) sum_j P_lj U_bj. Bound by the
// shared-memory reads of the two N-long products; P_lj is read as conj(P_jl) so
// that a warp's reads are consecutive.
template <int N>
struct ObsEl {
  static constexpr int KO = N == 8 ? 4 : 2;
  static constexpr int THREADS = KO * N * N;
};

template <int N>
__global__ void __launch_bounds__(ObsEl<N>::THREADS) k_obs_el(DevTables tb, const DevConsts* __restrict__ cst, ObsArgs a) {
  constexpr int NT = Tri<N>::NT, NN = N * N, KO = ObsEl<N>::KO, NW = ObsEl<N>::THREADS / 32;
  constexpr int NS = 3 * kPerX;
  __shared__ double2 sP[NN][KO], sH[NN][KO], sU[NN][KO];
  __shared__ double sTerm[NN][KO];
  __shared__ double sW[NW][NS];
  __shared__ double sPop[N][KO], sMax[N][KO], sMin[N][KO];
  __shared__ double sT[kFields];
  const int tid = threadIdx.x, kl = tid % KO, q = tid / KO, b = q / N, l = q % N;
  const int nk = tb.nk;
  const bool lower = b > l;
  const int e = lower ? Tri<N>::idx(l, b) : Tri<N>::idx(b, l);
  double acc[NS];
#pragma unroll
  for (int s = 0; s < NS; s++) acc[s] = 0.;
  double pop = 0., pmax = 0., pmin = 1.;
  const double2* rho = a.rho;
  const double2* hr = a.hr;
  const double2* U = hr ? a.uev : tb.U;
  pdl_wait();
  if (a.dyn && !a.dyn->obs_now) return;
  const int k1 = min((blockIdx.x + 1) * a.per * KO, nk);
  for (int k0 = blockIdx.x * a.per * KO; k0 < k1; k0 += KO) {
    const int k = k0 + kl;
    const bool valid = k < nk;
    const size_t o = (size_t)e * nk + k;
    double2 p = cz(), h = cz(), u = cz(), d[3] = {cz(), cz(), cz()};
    if (valid) {
      p = rho[o];
      h = (hr ? hr : tb.H)[o];
      u = U[(size_t)q * nk + k];
#pragma unroll
      for (int x = 0; x < 3; x++) {
        d[x] = tb.D[(size_t)x * NT * nk + o];
        if (lower && tb.herm_dip) d[x] = cconj(d[x]);
      }
      if (!lower) {
        if (a.want_current) {
          double2 ge[3] = {cz(), cz(), cz()};
          if (hr) {
            for (int bb = 0; bb < tb.nnb; bb++) {
              const double2 dh = csub(hr[(size_t)e * nk + tb.nbr[(size_t)bb * nk + k]], h);
#pragma unroll
              for (int x = 0; x < 3; x++) ge[x] = cadd(ge[x], cscale(dh, cst->wb[bb] * cst->bvec[bb][x]));
            }
          } else {
#pragma unroll
            for (int x = 0; x < 3; x++) ge[x] = tb.GE[(size_t)x * NT * nk + o];
          }
#pragma unroll
          for (int x = 0; x < 3; x++) {
            double2 j = cmul(p, ge[x]);
            if (b != l) j = cadd(j, cmul(cconj(p), cconj(ge[x])));
            acc[kPerX * x] += j.x;
            acc[kPerX * x + 1] += j.y;
          }
        }
        if (a.want_tabs && b < tb.nch && l >= tb.nch)
#pragma unroll
          for (int x = 0; x < 3; x++) {
            const double2 ta = cmul(cscale(d[x], 2.), p);
            acc[kPerX * x + 3] -= ta.x;
            acc[kPerX * x + 4] -= ta.y;
          }
      } else {
        p = cconj(p);
        h = cconj(h);
      }
#pragma unroll
      for (int x = 0; x < 3; x++) {
        const double2 pl = cmul(d[x], p);
        acc[kPerX * x + 5] += pl.x;
        acc[kPerX * x + 6] += pl.y;
      }
    }
    sP[q][kl] = p;
    sH[q][kl] = h;
    sU[q][kl] = u;
    __syncthreads();
    if (a.want_current) {
      double2 Q = cz();
#pragma unroll
      for (int i = 0; i < N; i++) Q = cadd(Q, cmul(sP[i * N + b][kl], sH[i * N + l][kl]));
#pragma unroll
      for (int x = 0; x < 3; x++) acc[kPerX * x + 2] += cmulc(Q, d[x]).y;
    }
    double2 m = cz();
#pragma unroll
    for (int j = 0; j < N; j++) m = cadd(m, cmul(cconj(sP[j * N + l][kl]), sU[b * N + j][kl]));
    sTerm[q][kl] = cmul(cconj(u), m).x;
    __syncthreads();
    if (valid && l == 0) {
      double pk = 0.;
#pragma unroll
      for (int j = 0; j < N; j++) pk += sTerm[b * N + j][kl];
      pop += pk;
      const double dev = b < tb.nbands ? 1. - pk : pk;
      pmax = fmax(pmax, fabs(dev));
      pmin = fmin(pmin, dev);
    }
  }
#pragma unroll
  for (int s = 0; s < NS; s++) {
    double x = acc[s];
    for (int w = 16; w > 0; w >>= 1) x += __shfl_xor_sync(0xffffffffu, x, w);
    if (tid % 32 == 0) sW[tid / 32][s] = x;
  }
  if (l == 0) {
    sPop[b][kl] = pop;
    sMax[b][kl] = pmax;
    sMin[b][kl] = pmin;
  }
  __syncthreads();
  double* part = a.part + blockIdx.x;
  const size_t np = gridDim.x;
  if (tid < NS) {
    double x = 0.;
    for (int w = 0; w < NW; w++) x += sW[w][tid];
    part[(kFX + tid) * np] = x;
  } else if (tid >= 32 && tid < 32 + N) {
    double x = 0.;
    for (int j = 0; j < KO; j++) x += sPop[tid - 32][j];
    part[(tid - 32) * np] = x;
  } else if (tid == 64 || tid == 65) {
    double x = tid == 64 ? 0. : 1.;
    for (int c = 0; c < N; c++)
      for (int j = 0; j < KO; j++) x = tid == 64 ? fmax(x, sMax[c][j]) : fmin(x, sMin[c][j]);
    part[(tid == 64 ? kFMax : kFMin) * np] = x;
  }
  obs_finish<N>(tb, a, sT);
}

// Rows U[c][i] = conj(Z[i][c]) of the eigenvectors of hr at every k: out[n * n][nk].
// WAVE: disjoint rotations together (eig.cuh).
template <int N, bool WAVE>
__global__ void __launch_bounds__(128) k_eig_rows(int nk, const double2* __restrict__ hr, double2* __restrict__ out,
                                                  const DynStep* __restrict__ dyn) {
  constexpr int LD = EigGroup<N>::LD, M = 128 / N;
  extern __shared__ double2 sm[];
  const int m = threadIdx.x / N, r = threadIdx.x % N, k0 = blockIdx.x * M;
  pdl_wait();
  if (dyn && !dyn->obs_now) return;
  for (int t = threadIdx.x; t < M * N * N; t += 128) {
    const int mk = t % M, ij = t / M, i = ij / N, j = ij % N;
    if (i > j) continue;
    const double2 v = hr[(size_t)Tri<N>::idx(i, j) * nk + min(k0 + mk, nk - 1)];
    double2* B = sm + mk * EigGroup<N>::WORDS;
    B[i * LD + j] = v;
    B[j * LD + i] = cconj(v);
  }
  __syncthreads();
  double2* A = sm + m * EigGroup<N>::WORDS;
  if (WAVE)
    eig_herm_wave<N>(A, A + N * LD, r);
  else
    eig_herm_group<N>(A, A + N * LD, r);
  __syncthreads();
  for (int t = threadIdx.x; t < M * N * N; t += 128) {
    const int mk = t % M, ij = t / M, i = ij / N, j = ij % N;
    if (k0 + mk < nk) out[(size_t)ij * nk + k0 + mk] = cconj(sm[mk * EigGroup<N>::WORDS + N * LD + j * LD + i]);
  }
}

template <int N>
cudaError_t launch_obs_n(const DevTables& tb, const DevConsts* cst, const ObsArgs& a, cudaStream_t s) {
  return launch_pdl(k_obs<N>, dim3((tb.nk + kObsThreads - 1) / kObsThreads), dim3(kObsThreads), 0, s, tb, cst, a);
}

template <int N>
cudaError_t launch_obs_el(const DevTables& tb, const DevConsts* cst, ObsArgs a, double2* uev, bool coulomb, cudaStream_t s) {
  if (a.hr) {
    if (!uev) return cudaErrorInvalidValue;
    constexpr int M = 128 / N;
    constexpr size_t smem = sizeof(double2) * EigGroup<N>::WORDS * M;
    cudaError_t e = cudaSuccess;
    auto eig = coulomb ? k_eig_rows<N, false> : k_eig_rows<N, true>;
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(eig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = launch_pdl(eig, dim3((tb.nk + M - 1) / M), dim3(128), smem, s, tb.nk, a.hr, uev, a.dyn);
    if (e != cudaSuccess) return e;
    a.uev = uev;
  }
  const int subs = (tb.nk + ObsEl<N>::KO - 1) / ObsEl<N>::KO;
  a.per = (subs + kObsElBlocks - 1) / kObsElBlocks;
  return launch_pdl(k_obs_el<N>, dim3((subs + a.per - 1) / a.per), dim3(ObsEl<N>::THREADS), 0, s, tb, cst, a);
}

}  // namespace

int obs_parts(int nk) {
  const int b = (nk + kObsThreads - 1) / kObsThreads;
  return b > kObsElBlocks ? b : kObsElBlocks;
}
size_t obs_part_bytes() { return sizeof(ObsPart); }
size_t obs_eig_count(int n, int nk) { return n >= 8 ? (size_t)n * n * nk : 0; }

cudaError_t launch_observables(const DevTables& tb, const DevConsts* cst, const double2* rho, const double2* hr, bool coulomb, double2* uev,
                               int want_current, int want_tabs, void* part, unsigned int* done, double scaleJ,
                               double scaleTA, const ObsRecord& rec, ObsRecord* log, double* ncond_dev,
                               double* pcmax_dev, cudaStream_t s, const DynStep* dyn) {
  ObsArgs a;
  a.dyn = dyn;
  a.rho = rho;
  a.hr = hr;
  a.uev = nullptr;
  a.per = 0;
  a.want_current = want_current;
  a.want_tabs = want_tabs && tb.nch > 0;
  a.part = (double*)part;
  a.done = done;
  a.scaleJ = scaleJ;
  a.scaleTA = scaleTA;
  a.rec = rec;
  a.log = log;
  a.ncond_dev = ncond_dev;
  a.pcmax_dev = pcmax_dev;
  switch (tb.n) {
    case 1: return launch_obs_n<1>(tb, cst, a, s);
    case 2: return launch_obs_n<2>(tb, cst, a, s);
    case 3: return launch_obs_n<3>(tb, cst, a, s);
    case 4: return launch_obs_n<4>(tb, cst, a, s);
    case 5: return launch_obs_n<5>(tb, cst, a, s);
    case 8: return launch_obs_el<8>(tb, cst, a, uev, coulomb, s);
    case 16: return launch_obs_el<16>(tb, cst, a, uev, coulomb, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace edus
