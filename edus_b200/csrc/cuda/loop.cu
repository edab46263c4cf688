// loop.cu — a whole constant-dt solve (RK4 or Adams-Bashforth, FP64) in one
// launch, for grids that fit the GPU at one thread per (k point, element).
//
// The launch per stage (rhs_ep.cu) of such a solve is latency: 3.7 us a stage for
// 24 x 24 hBN, where the arithmetic of a stage is 0.1 us, since every launch loads
// its tables, its own state and the stencil's indices again before it can start.
// Here a block keeps KT k points for the whole run: state, stage accumulator, H
// and the Adams-Bashforth history stay in registers, dipoles and stencil indices
// in shared memory; only the stage input goes through global memory (L2), because
// the k-gradient reads other blocks' k points. Stages are separated by a barrier
// over the blocks. Output instants are taken by the same blocks between two
// barriers; one more block adds up their partials while the others step on.
// A stage is then about 2.7 us (60 x 60): the barrier 1.4 us (one release, one
// atomic and a poll through L2; an array of flags polled by every block took 2.4),
// stencil gathers 0.4, the element's own work 0.8.
//   60 x 60 hBN, RK4, a record every step: 14.8 us a step, 28.7 before
//   24 x 24 hBN, RK4 (one cluster): 6.7 us a step, 13.8 before
//   70 x 70 with core-hole decay, AB5: 5.5 us a step, 10.5 before
//
// The blocks wait on one another, so the launch is cooperative (all blocks
// resident) or one cluster. A wait on the cooperative grid is bounded and records
// kErrTimeout; the cluster's hardware barrier has no bound: its blocks are placed
// together and make the same barrier calls. Data written by other blocks is read past L1.
//
// Arithmetic: every element goes through the expressions of k_rhs_ep in the same
// order, but for relaxation, whose products are formed once per k point.
#include <algorithm>
#include <type_traits>

#include "dev.cuh"
#include "eig.cuh"
#include "kernels.hpp"
#include "loop.cuh"
#include "obs.cuh"

namespace edus {
namespace {

template <int N>
struct TriL {
  static constexpr int NT = N * (N + 1) / 2;
  static __device__ __forceinline__ int idx(int i, int j) { return i * N - (i * (i - 1)) / 2 + (j - i); }
  static __device__ __forceinline__ void ij(int e, int& i, int& j) {
    int r = e;
    i = 0;
    while (r >= N - i) {
      r -= N - i;
      i++;
    }
    j = i + r;
  }
};

// Most threads of a block: 168 registers each, or 96 for the largest grids, which spill
// (3 bands 340 bytes, 5 bands 400).
constexpr int kLoopSmall = 384, kLoopThreads = 640;
constexpr int kSumF = 3 * kPerX;   // current fields of a block partial

// Polls of a grid barrier before it gives up, tens of seconds: at a launch's first
// barrier the last blocks may still wait for room that another program's kernels hold.
constexpr int kGridWaitIters = 1 << 26;

__host__ __device__ constexpr size_t pad16(size_t b) { return (b + 15) & ~(size_t)15; }

// Dynamic shared memory of a block of at most MAXT threads. Planes over the
// block's k points have the compile-time stride KS.
template <int N, int MAXT>
struct LoopSmem {
  static constexpr int NT = TriL<N>::NT, KS = MAXT / NT;
  double2 *sP, *sH, *sD, *sU, *sM;  // sP, sH, sU, sM: full matrices [N * N][KS]
  double *sPop, *sGc;
  int* sN;
  LoopStep* sS;
  double2* sX;  // cluster: stage inputs that the other blocks read, [2][NT][KS]
  size_t bytes;
  __host__ __device__ LoopSmem(unsigned char* base, const DevTables& tb, int nb, int ngc, int ncomp, bool cluster) {
    size_t off = 0;
    auto take = [&](size_t b) {
      unsigned char* r = base + off;
      off += pad16(b);
      return r;
    };
    sP = (double2*)take(sizeof(double2) * N * N * KS);
    sH = (double2*)take(sizeof(double2) * N * N * KS);
    sD = (double2*)take(sizeof(double2) * NT * KS * ncomp);
    sU = (double2*)take(tb.n_diss > 0 ? sizeof(double2) * N * N * KS : 0);
    sM = (double2*)take(tb.n_diss > 0 ? sizeof(double2) * N * N * KS : 0);
    sPop = (double*)take(sizeof(double) * N * KS);
    sGc = (double*)take(sizeof(double) * 2 * ngc);
    sN = (int*)take(sizeof(int) * nb * KS);
    sS = (LoopStep*)take(2 * sizeof(LoopStep));
    sX = (double2*)take(cluster ? sizeof(double2) * 2 * NT * KS : 0);
    bytes = off;
  }
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Entry off (in double2) of block rank's copy of the shared array at base.
__device__ __forceinline__ double2 ld_cluster(uint32_t base, int rank, int off) {
  uint32_t at;
  double2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at + 16u * (uint32_t)off) : "memory");
  return v;
}

// Barrier over all blocks; false when the bounded wait ran out (the same for
// every thread of a block). On a cluster the hardware barrier, with release and
// acquire of the blocks' global writes.
struct GridBar {
  unsigned int* ctr;
  unsigned int target, blocks;
  int* err;
  bool cluster;
  bool* ok;  // shared
  __device__ bool sync() {
    if (cluster) {
      asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
      return true;
    }
    __syncthreads();
    target += blocks;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      bool got = false;
      for (int it = 0; it < kGridWaitIters; ++it) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if ((int)(v - target) >= 0) {
          got = true;
          break;
        }
      }
      if (!got) atomicExch(err, kErrTimeout);
      *ok = got;
    }
    __syncthreads();
    return *ok;
  }
};

// Sums of M values (a power of two, at most 8) over the warp: lane l (l < M)
// returns the sum of value l. Halving exchange: 2 M shuffles fewer than a
// butterfly per value.
template <int M>
__device__ __forceinline__ double warp_sums(double (&v)[M]) {
  const int lane = threadIdx.x % 32;
#pragma unroll
  for (int h = M / 2; h > 0; h >>= 1) {
    const bool up = lane & h;
#pragma unroll
    for (int q = 0; q < h; q++) {
      const double keep = up ? v[q + h] : v[q], give = up ? v[q] : v[q + h];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, h);
    }
  }
  double x = v[0];
#pragma unroll
  for (int s = M; s < 32; s <<= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
  return x;
}

// CL: one cluster, the stage inputs exchanged through distributed shared memory
// and written to global memory in the last step only. The barrier's release has
// then no global stores to wait for (0.28 us for 0.9) and a gather is a read
// of another SM's shared memory, not of L2. 24 x 24 hBN, RK4: 6.7 us a step, 8.0
// with the exchange through L2.
template <int N, bool AB, int MAXT, bool CL>
__global__ void __launch_bounds__(MAXT) k_loop(const __grid_constant__ LoopArgs a) {
  constexpr int NT = TriL<N>::NT, KS = MAXT / NT;
  const DevTables& tb = a.tb;
  extern __shared__ __align__(16) unsigned char loop_smem_raw[];
  const int kt = a.kt, nk = tb.nk, nb = a.nb_sel, npc = a.npc, nbp = a.nbp, ngc = a.ngc;
  const int ncomp = a.ncomp;
  const LoopSmem<N, MAXT> S(loop_smem_raw, tb, nb, ngc, ncomp, CL);
  __shared__ double sW[MAXT / 32][33];
  __shared__ double sT[kFields];
  __shared__ bool sOk;
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid % 32, warp = tid / 32, nwarp = nthr / 32;
  const int nstep_blocks = gridDim.x - 1;
  const bool stepper = (int)blockIdx.x < nstep_blocks;
  GridBar bar{a.bar, 0u, gridDim.x, tb.err, CL, &sOk};

  // ---------------------------------------------------------- the adding block
  // Joins every barrier; after the first one behind an instant the partials are
  // complete, and they are added while the others take the next stage. Partials
  // are double buffered by instant, so the next instant never overwrites them.
  if (!stepper) {
    constexpr int kF = kSumF + N + 2;  // fields of a partial: currents, populations, max, min
    static_assert(kF <= 32, "a partial is one 32-word row");
    int inst = 0;
    if (CL) bar.sync();  // the first stage inputs
    for (int it = 0; it < a.nsteps; it++) {
      const bool obs = (a.it0 + it) % a.res == 0;
      const int nbar = AB && a.it0 + it >= a.nstartup ? 1 : 4;
      for (int q = 0; q < nbar; q++) {
        if (!bar.sync()) return;
        if (!obs || q != 0) continue;
        // block partials: a warp per slice of the blocks, a lane per field
        const double* part = a.part + (size_t)(inst & 1) * 32 * nstep_blocks;
        double x = lane == kF - 1 ? 1. : 0.;
        if (lane < kF)
          for (int b0 = warp; b0 < nstep_blocks; b0 += 8 * nwarp) {
            double y[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
              y[u] = b0 + u * nwarp < nstep_blocks ? __ldcg(part + (size_t)(b0 + u * nwarp) * 32 + lane) : (lane == kF - 1 ? 1. : 0.);
#pragma unroll
            for (int u = 0; u < 8; u++) x = lane == kF - 2 ? fmax(x, y[u]) : (lane == kF - 1 ? fmin(x, y[u]) : x + y[u]);
          }
        sW[warp][lane] = x;
        __syncthreads();
        if (warp == 0 && lane < kF) {
          for (int w = 1; w < nwarp; w++) {
            const double y = sW[w][lane];
            x = lane == kF - 2 ? fmax(x, y) : (lane == kF - 1 ? fmin(x, y) : x + y);
          }
          const int f = lane < kSumF ? kFX + lane : (lane < kSumF + N ? lane - kSumF : (lane == kF - 2 ? kFMax : kFMin));
          sT[f] = x;
        }
        __syncthreads();
        if (warp == 0 && inst < a.log_cap) {
          // the record, its parts on different lanes (obs_fill's formulas)
          const LoopStep* st = reinterpret_cast<const LoopStep*>(a.steps + (size_t)it * a.stride);
          ObsRecord* rec = a.log + inst;
          const double inv = 1. / nk;
          if (lane < 3) {
            const double* f = sT + kFX + kPerX * lane;
            rec->J1[2 * lane] = f[0] * a.scaleJ;
            rec->J1[2 * lane + 1] = f[1] * a.scaleJ;
            rec->J2[lane] = -2. * (f[2] * a.scaleJ);
            rec->tabs[2 * lane] = f[3] * a.scaleTA * inv;
            rec->tabs[2 * lane + 1] = f[4] * a.scaleTA * inv;
            rec->pol[2 * lane] = f[5] * inv;
            rec->pol[2 * lane + 1] = f[6] * inv;
          } else if (lane == 3) {
            double trace = -(double)tb.nbands, nc = 0;
            for (int c = 0; c < N; c++) {
              const double v = sT[c] * inv, p = c < tb.nbands ? 1.0 - v : v;
              trace += v;
              if (p > nc) nc = p;
            }
            rec->trace_dev = trace;
            rec->n_cond = nc;
            rec->p_cond_max = sT[kFMax];
            rec->p_min = sT[kFMin];
            *a.ncond_dev = nc;
            *a.pcmax_dev = sT[kFMax];
          } else if (lane == 4) {
            rec->t = st->t;
            rec->dt = a.dt;
          } else if (lane < 8) {
            rec->EF_pump[lane - 5] = st->EF_last[0][lane - 5];
            rec->EF_probe[lane - 5] = st->EF_last[1][lane - 5];
          } else if (lane < 8 + kMaxBands) {
            const int c = lane - 8;
            const double v = c < N ? sT[c] * inv : 0.;
            rec->pop[c] = c < N && c < tb.nbands ? 1.0 - v : v;
          }
        }
        __syncthreads();
        inst++;
      }
    }
    return;
  }

  // ---------------------------------------------------------- set-up
  const int kl = tid % kt, e = tid / kt;  // threads past NT * kt only help with shared work
  const int k = blockIdx.x * kt + kl;
  const bool own = e < NT;
  const bool valid = own && k < nk;
  int i = 0, j = 0;
  if (own) TriL<N>::ij(e, i, j);
  const size_t o = (size_t)(own ? e : 0) * nk + (k < nk ? k : 0);
  double2 Pe = cz(), He = cz(), acc = cz();
  if (valid) {
    Pe = a.P0[o];
    He = tb.H[o];
    for (int c = 0; c < ncomp; c++) S.sD[(c * NT + e) * KS + kl] = tb.D[(size_t)a.comp[c] * NT * nk + o];
  }
  double2 R[AB ? 4 : 1];  // previous derivatives, newest first
#pragma unroll
  for (int q = 0; q < (AB ? 4 : 1); q++) R[q] = AB && valid && q < a.order - 1 ? a.ring[(size_t)q * NT * nk + o] : cz();
  if (tb.n_diss > 0)
    for (int t = tid; t < N * N * kt; t += nthr) S.sU[(t / kt) * KS + t % kt] = tb.U[(size_t)(t / kt) * nk + min((int)(blockIdx.x * kt) + t % kt, nk - 1)];
  for (int t = tid; t < nb * kt; t += nthr)
  {
    const int kb = tb.nbr[(size_t)a.bsel[t / kt] * nk + min((int)(blockIdx.x * kt) + t % kt, nk - 1)];
    S.sN[(t / kt) * KS + t % kt] = CL ? (kb / kt) << 16 | kb % kt : kb;  // CL: block and place
  }
  const uint32_t xbase = smem_u32(S.sX);
  if (CL && valid) S.sX[e * KS + kl] = Pe;
  // step record it and its gradient coefficients into buffer it & 1, asynchronously
  auto fetch = [&](int it) {
    if (it < a.nsteps) {
      constexpr int kWords = sizeof(LoopStep) / 16;
      const int4* src = reinterpret_cast<const int4*>(a.steps + (size_t)it * a.stride);
      if (tid < kWords) cp_async16(reinterpret_cast<int4*>(S.sS + (it & 1)) + tid, src + tid);
      for (int t = tid; t < ngc / 2; t += nthr) cp_async16(reinterpret_cast<int4*>(S.sGc + (it & 1) * ngc) + t, src + kWords + t);
    }
  };
  auto fetched = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
  // relaxation pairs and rates: in global memory they were two dependent reads a
  // pair past an L1 that every grid barrier empties, 1800 cycles a stage
  __shared__ int sRel[N * N];
  __shared__ double sRelT[N * N];
  for (int t = tid; t < tb.n_diss; t += nthr) {
    sRel[t] = a.cst->diss_i[t] * N + a.cst->diss_j[t];
    sRelT[t] = a.cst->T[sRel[t]];
  }
  fetch(0);
  fetched();
  if (CL)
    bar.sync();
  else
    __syncthreads();
  double2 tii = cz();  // relaxation towards the filled bands: constant
  if (tb.n_diss > 0 && valid)
    for (int q = 0; q < tb.nbands; q++)
      tii = cadd(tii, cscale(cmulc(S.sU[(q * N + i) * KS + kl], S.sU[(q * N + j) * KS + kl]), a.cst->T[q * N + q]));
  // stage input kb of this element: from L2, or from the block that owns it
  int xb = 0;  // CL: half of sX with the stage inputs
  auto input = [&](const double2* src, int kb) {
    if constexpr (CL) return ld_cluster(xbase, kb >> 16, (xb * NT + e) * KS + (kb & 0xFFFF));
    else return __ldcg(src + (size_t)e * nk + kb);
  };
  double2* cur = a.P0;   // buffer of the current state
  double2* oth = a.Pa;
  int inst = 0;
  const bool herm = tb.herm_dip != 0;
  auto Pf = [&](int r, int c) -> double2 { return S.sP[(r * N + c) * KS + kl]; };
  auto HF = [&](int r, int c) -> double2 { return S.sH[(r * N + c) * KS + kl]; };
  // full matrices of this k point from its upper elements: P, and H with its lower entry hl
  auto publish = [&](double2 p, double2 hu, double2 hl) {
    S.sP[(i * N + j) * KS + kl] = p;
    S.sH[(i * N + j) * KS + kl] = hu;
    if (i != j) {
      S.sP[(j * N + i) * KS + kl] = cconj(p);
      S.sH[(j * N + i) * KS + kl] = hl;
    }
  };

  for (int it = 0; it < a.nsteps; it++) {
    const LoopStep& st = S.sS[it & 1];
    const double* gco = S.sGc + (it & 1) * ngc;
    fetch(it + 1);

    // -------------------------------------------------------- output instant
    if (st.obs) {
      // the tables of an instant in flight first
      double2 ge[3] = {cz(), cz(), cz()}, dd[3] = {cz(), cz(), cz()}, Uc[N];
      if (valid) {
#pragma unroll
        for (int x = 0; x < 3; x++) {
          dd[x] = tb.D[(size_t)x * NT * nk + o];
          if (a.want_current) ge[x] = tb.GE[(size_t)x * NT * nk + o];
        }
      }
      if (e < N && k < nk) {
#pragma unroll
        for (int q = 0; q < N; q++) Uc[q] = tb.U[(size_t)(e * N + q) * nk + k];
      }
      if (own) publish(Pe, He, cconj(He));
      __syncthreads();
      if (e < N) {
        const int c = e;
        double Pik = 0.;
        if (k < nk) {
          double2 pa = cz();
#pragma unroll
          for (int ii = 0; ii < N; ii++) {
            double2 m = cz();
#pragma unroll
            for (int jj = 0; jj < N; jj++) m = cadd(m, cmul(Pf(ii, jj), Uc[jj]));
            pa = cadd(pa, cmul(cconj(Uc[ii]), m));
          }
          Pik = pa.x;
        }
        S.sPop[c * KS + kl] = Pik;
      }
      double2 J1[3] = {cz(), cz(), cz()}, PL[3], TA[3] = {cz(), cz(), cz()};
      double J2[3] = {0., 0., 0.};
#pragma unroll
      for (int x = 0; x < 3; x++) PL[x] = cz();
      if (valid) {
        if (a.want_current) {
#pragma unroll
          for (int x = 0; x < 3; x++) {
            J1[x] = cmul(Pe, ge[x]);
            if (i != j) J1[x] = cadd(J1[x], cmul(cconj(Pe), cconj(ge[x])));
          }
        }
        double2 Q0 = cz(), Q1 = cz();
        if (a.want_current)
          for (int q = 0; q < N; q++) {
            Q0 = cadd(Q0, cmul(Pf(q, i), HF(q, j)));
            Q1 = cadd(Q1, cmul(Pf(q, j), HF(q, i)));
          }
#pragma unroll
        for (int x = 0; x < 3; x++) {
          const double2 d = dd[x], dl = herm ? cconj(d) : d;
          PL[x] = cmul(d, Pe);
          if (a.want_current) J2[x] = cmulc(Q0, d).y;
          if (i != j) {
            PL[x] = cadd(PL[x], cmul(dl, cconj(Pe)));
            if (a.want_current) J2[x] += cmulc(Q1, dl).y;
          }
          if (a.want_tabs && i < tb.nch && j >= tb.nch) TA[x] = csub(TA[x], cmul(cscale(d, 2.), Pe));
        }
      }
      double v0[8] = {J1[0].x, J1[0].y, J1[1].x, J1[1].y, J1[2].x, J1[2].y, J2[0], J2[1]};
      double v1[8] = {PL[0].x, PL[0].y, PL[1].x, PL[1].y, PL[2].x, PL[2].y, J2[2], 0.};
      const double s0 = warp_sums<8>(v0), s1 = warp_sums<8>(v1);
      double s2 = 0.;
      if (a.want_tabs) {
        double v2[8] = {TA[0].x, TA[0].y, TA[1].x, TA[1].y, TA[2].x, TA[2].y, 0., 0.};
        s2 = warp_sums<8>(v2);
      }
      if (lane < 6) {
        const int x = lane / 2, m = lane % 2;
        sW[warp][kPerX * x + m] = s0;
        sW[warp][kPerX * x + 5 + m] = s1;
        sW[warp][kPerX * x + 3 + m] = s2;
      } else if (lane == 6) {
        sW[warp][2] = s0;
        sW[warp][kPerX * 2 + 2] = s1;
      } else if (lane == 7) {
        sW[warp][kPerX + 2] = s0;
      }
      __syncthreads();
      double* part = a.part + ((size_t)(inst & 1) * nstep_blocks + blockIdx.x) * 32;
      if (tid < kSumF) {
        double x = 0.;
        for (int w = 0; w < nwarp; w++) x += sW[w][tid];
        __stcg(part + tid, x);
      }
      // populations: band sums and the extremes of all bands, a warp each (the last
      // warps; the first adds up the currents)
      const int left = nk - blockIdx.x * kt, kn = left < kt ? left : kt;
      for (int task = nwarp - 1 - warp; task <= N; task += nwarp) {
        if (task < N) {
          double x = 0.;
          for (int q = lane; q < kn; q += 32) x += S.sPop[task * KS + q];
          for (int s = 16; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
          if (lane == 0) __stcg(part + kSumF + task, x);
        } else {
          double lo = 1., hi = 0.;
          for (int c = 0; c < N; c++)
            for (int q = lane; q < kn; q += 32) {
              const double p = S.sPop[c * KS + q], dev = c < tb.nbands ? 1. - p : p;
              hi = fmax(hi, fabs(dev));
              lo = fmin(lo, dev);
            }
          for (int s = 16; s > 0; s >>= 1) {
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, s));
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, s));
          }
          if (lane == 0) {
            __stcg(part + kSumF + N, hi);
            __stcg(part + kSumF + N + 1, lo);
          }
        }
      }
      __syncthreads();
      inst++;
    }

    // -------------------------------------------------------- stages of the step
    const bool rk = !AB || st.startup;
    const int nstage = rk ? 4 : 1;
    double2 pin = Pe;
    const double2* src = cur;
    const bool last = it == a.nsteps - 1;
    // the next stage's input, read by the other blocks behind the barrier
    auto hand = [&](double2* dst, double2 x) {
      if (CL) S.sX[((xb ^ 1) * NT + e) * KS + kl] = x;
      if (!CL || last) dst[o] = x;
    };
    for (int sg = 0; sg < nstage; sg++) {
      const int fi = sg == 0 ? 0 : (sg == 3 ? 2 : 1);
      // stencil gathers in flight before the element's own work
      constexpr int NG = MAXT <= kLoopSmall ? 12 : 6;  // hexagonal and square grids have up to 12
      double2 pn[NG];
      const bool grad = st.e_non0 && valid;
#pragma unroll
      for (int c = 0; c < NG; c++) pn[c] = grad && c < nb ? input(src, S.sN[c * KS + kl]) : cz();
      if (own) {
        const int w = (i < tb.nch) != (j < tb.nch);
        double2 hu = He, hl = cconj(He);
        for (int c = 0; c < ncomp; c++) {
          const double f = st.EF[fi][w][a.comp[c]];
          const double2 d = S.sD[(c * NT + e) * KS + kl];
          hu = cadd(hu, cscale(d, f));
          hl = cadd(hl, cscale(herm ? cconj(d) : d, f));
        }
        publish(pin, hu, hl);
      }
      __syncthreads();
      if (tb.n_diss > 0) {
        if (valid) {
          double2 m = cz();
#pragma unroll
          for (int q = 0; q < N; q++) {
            double2 w = cz();
#pragma unroll
            for (int p = 0; p < N; p++) w = cadd(w, cmulc(Pf(p, q), S.sU[(i * N + p) * KS + kl]));
            m = cadd(m, cmul(S.sU[(j * N + q) * KS + kl], w));
          }
          S.sM[(i * N + j) * KS + kl] = m;
          if (i != j) S.sM[(j * N + i) * KS + kl] = cconj(m);
        }
        __syncthreads();
      }
      if (valid) {
        double2 v;
        if (i == j) {
          double2 beta = cz();
#pragma unroll
          for (int l = 0; l < N; l++) beta = cadd(beta, cmul(HF(i, l), Pf(i, l)));
          v = cmk(2. * beta.y, 0.);
        } else {
          double2 beta = cz();
#pragma unroll
          for (int l = 0; l < N; l++) {
            const double2 x = cmul(HF(j, l), Pf(i, l));
            const double2 y = cmul(HF(i, l), Pf(j, l));
            beta = cadd(beta, csub(x, cconj(y)));
          }
          v = cmi(beta);
          if (i < tb.nch && j >= tb.nch) v = cadd(v, cmi(cscale(pin, -a.wx2)));
        }
        if (tb.n_diss > 0) {
          // M = conj(U) P U^T is formed once per k point (k_rhs_ep's threads each form
          // every M they use)
          for (int t = 0; t < tb.n_diss; t++) {
            const int ii = sRel[t] / N, jj = sRel[t] % N;
            const double2 f = cscale(cmulc(cconj(S.sU[(jj * N + j) * KS + kl]), S.sU[(i * N + ii) * KS + kl]), sRelT[t]);
            v = csub(v, cmul(f, S.sM[(ii * N + jj) * KS + kl]));
          }
          v = cadd(v, tii);
        }
        double2 G = cz();
        if (grad) {
          const double* g = gco + fi * npc * nbp;
          auto add = [&](const double2* p, int c0, auto count) {  // (coefficients are zero past nb)
            if (npc == 1) {
#pragma unroll
              for (int c = 0; c < count(); c++) G = cadd(G, cscale(p[c], g[c0 + c]));
            } else {
#pragma unroll
              for (int c = 0; c < count(); c++)
                for (int x = 0; x < npc; x++) G = cadd(G, cscale(p[c], g[x * nbp + c0 + c]));
            }
          };
          add(pn, 0, std::integral_constant<int, NG>());
          for (int c0 = NG; c0 < nb; c0 += 6) {
            double2 p[6];
#pragma unroll
            for (int c = 0; c < 6; c++) p[c] = c0 + c < nb ? input(src, S.sN[(c0 + c) * KS + kl]) : cz();
            add(p, c0, std::integral_constant<int, 6>());
          }
        }
        v = cadd(v, G);
        if (i == j) v.y = 0.;
        if (rk) {
          if (sg == 0) {
            if (AB) {
#pragma unroll
              for (int q = 3; q > 0; q--) R[AB ? q : 0] = R[AB ? q - 1 : 0];
              R[0] = v;
            }
            acc = cadd(Pe, cscale(v, a.dt6));
            pin = cadd(Pe, cscale(v, a.dt2));
            hand(oth, pin);
          } else if (sg < 3) {
            acc = cadd(acc, cscale(v, a.dt3));
            pin = cadd(Pe, cscale(v, sg == 1 ? a.dt2 : a.dt));
            hand(sg == 1 ? a.Pb : oth, pin);
            if (sg == 2 && (AB || last)) a.P1[o] = acc;
          } else {
            Pe = cadd(acc, cscale(v, a.dt6));
            hand(cur, Pe);
          }
        } else if (AB) {
          double2 d = cz();
          d = cadd(d, cscale(v, a.coef[0]));
#pragma unroll
          for (int q = 1; q < 5; q++)
            if (q < a.order) d = cadd(d, cscale(R[AB ? q - 1 : 0], a.coef[q]));
#pragma unroll
          for (int q = 3; q > 0; q--) R[AB ? q : 0] = R[AB ? q - 1 : 0];
          R[0] = v;
          Pe = cadd(Pe, cscale(d, a.dt));
          hand(oth, Pe);
        }
      }
      xb ^= 1;
      if (rk) src = sg == 1 ? a.Pb : oth;
      if (sg == nstage - 1) fetched();
      if (!bar.sync()) return;
    }
    if (AB && !rk) {
      double2* t = cur;
      cur = oth;
      oth = t;
    }
  }
  if (AB && valid) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < a.order - 1) a.ring[(size_t)q * NT * nk + o] = R[AB ? q : 0];
  }
}

// Launch attributes of a plan, for the launch and for the question whether it fits.
template <int N, bool AB, int MAXT, bool CL>
struct LoopLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cudaError_t prepare(const LoopPlan& p, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_loop<N, AB, MAXT, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e == cudaSuccess && CL && p.blocks + 1 > 8)
      e = cudaFuncSetAttribute(k_loop<N, AB, MAXT, CL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cfg.gridDim = dim3(p.blocks + 1);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    if (CL) {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = p.blocks + 1;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return e;
  }
};

template <int N, bool AB, int MAXT, bool CL>
cudaError_t loop_launch_t(const LoopArgs& a, const LoopPlan& p, cudaStream_t s) {
  LoopLaunch<N, AB, MAXT, CL> l;
  const cudaError_t e = l.prepare(p, s);
  return e == cudaSuccess ? cudaLaunchKernelEx(&l.cfg, k_loop<N, AB, MAXT, CL>, a) : e;
}

// All blocks of the plan resident at once.
template <int N, bool AB, int MAXT, bool CL>
bool loop_fits_t(const LoopPlan& p, int sms) {
  LoopLaunch<N, AB, MAXT, CL> l;
  int n = 0;
  cudaError_t e = l.prepare(p, nullptr);
  if (e == cudaSuccess && CL) e = cudaOccupancyMaxActiveClusters(&n, k_loop<N, AB, MAXT, CL>, &l.cfg);
  if (e == cudaSuccess && !CL) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_loop<N, AB, MAXT, CL>, p.threads, p.smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return CL ? n >= 1 : (long long)n * sms >= p.blocks + 1;
}

template <int N, bool AB>
cudaError_t loop_launch(const LoopArgs& a, const LoopPlan& p, cudaStream_t s) {
  if (p.cluster) return p.small ? loop_launch_t<N, AB, kLoopSmall, true>(a, p, s) : cudaErrorInvalidValue;
  return p.small ? loop_launch_t<N, AB, kLoopSmall, false>(a, p, s) : loop_launch_t<N, AB, kLoopThreads, false>(a, p, s);
}

template <int N, bool AB>
bool loop_fits(const LoopPlan& p, int sms) {
  if (p.cluster) return p.small && loop_fits_t<N, AB, kLoopSmall, true>(p, sms);
  return p.small ? loop_fits_t<N, AB, kLoopSmall, false>(p, sms) : loop_fits_t<N, AB, kLoopThreads, false>(p, sms);
}

template <int N>
size_t loop_smem(const DevTables& tb, bool small, int nb, int ngc, int ncomp, bool cluster) {
  return small ? LoopSmem<N, kLoopSmall>(nullptr, tb, nb, ngc, ncomp, cluster).bytes
               : LoopSmem<N, kLoopThreads>(nullptr, tb, nb, ngc, ncomp, cluster).bytes;
}

bool loop_plan_fits(int n, bool ab, const LoopPlan& p, int sms) {
#define X(n) \
  case n: return ab ? loop_fits<n, true>(p, sms) : loop_fits<n, false>(p, sms);
  switch (n) {
    X(1) X(2) X(3) X(4) X(5)
    default: return false;
  }
#undef X
}

// One block per SM, one of them adding up the instants; a block of at least 128
// threads (with fewer a block, more blocks only lengthen the barrier) and at most
// 640. A grid that 15 such blocks of kLoopSmall threads hold runs as one cluster
// of up to 16 with the hardware barrier. Larger grids, the mean field (whose
// transforms are bound by shared memory, 24.4 us a step here against 22.2 with
// the launch per stage on 120 x 120) and 8 and 16 bands keep the launch per stage.
LoopPlan loop_shape(const DevTables& tb, int nb, int ngc, int ncomp, int sms, bool cluster) {
  LoopPlan p;
  if (tb.n < 1 || tb.n > 5 || tb.h || sms < 2) return p;
  const int nt = tb.ntri;
  const int kt_min = (128 + nt - 1) / nt;
  int blocks = std::min((tb.nk + kt_min - 1) / kt_min, sms - 1);
  p.cluster = cluster && (tb.nk + 14) / 15 <= kLoopSmall / nt;
  if (p.cluster) blocks = std::min(blocks, 15);
  p.kt = (tb.nk + blocks - 1) / blocks;
  blocks = (tb.nk + p.kt - 1) / p.kt;
  const int threads = (nt * p.kt + 31) / 32 * 32;
  if (threads > kLoopThreads || p.kt > kLoopThreads / nt || blocks < 1) return p;
  p.small = threads <= kLoopSmall && p.kt <= kLoopSmall / nt;
  switch (tb.n) {
    case 1: p.smem = loop_smem<1>(tb, p.small, nb, ngc, ncomp, p.cluster); break;
    case 2: p.smem = loop_smem<2>(tb, p.small, nb, ngc, ncomp, p.cluster); break;
    case 3: p.smem = loop_smem<3>(tb, p.small, nb, ngc, ncomp, p.cluster); break;
    case 4: p.smem = loop_smem<4>(tb, p.small, nb, ngc, ncomp, p.cluster); break;
    case 5: p.smem = loop_smem<5>(tb, p.small, nb, ngc, ncomp, p.cluster); break;
  }
  if (p.smem > 220 * 1024) return p;
  p.threads = threads;
  p.part = (size_t)2 * 32 * blocks;
  p.blocks = blocks;
  return p;
}

}  // namespace

// The first form whose blocks the device holds at once: it may not place so wide a
// cluster, or lend the process fewer SMs than it has.
LoopPlan loop_plan(const DevTables& tb, int nb, int ngc, int ncomp, int sms, bool ab) {
  LoopPlan p = loop_shape(tb, nb, ngc, ncomp, sms, true);
  if (p.blocks > 0 && p.cluster && !loop_plan_fits(tb.n, ab, p, sms)) p = loop_shape(tb, nb, ngc, ncomp, sms, false);
  if (p.blocks > 0 && !loop_plan_fits(tb.n, ab, p, sms)) p = LoopPlan();
  return p;
}

cudaError_t launch_loop(const LoopArgs& a, const LoopPlan& p, cudaStream_t s) {
  const bool ab = a.order > 0;
#define X(n) \
  case n: return ab ? loop_launch<n, true>(a, p, s) : loop_launch<n, false>(a, p, s);
  switch (a.tb.n) {
    X(1) X(2) X(3) X(4) X(5)
    default: return cudaErrorInvalidValue;
  }
#undef X
}

}  // namespace edus
